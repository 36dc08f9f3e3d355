// wfa_tiers.cu -- gap-affine WFA cost with the wavefront rings in shared memory.
//
// Computes wfa_affine_cpu (genomics/cpu/align_cpu.mojo:75-226) exactly, with
// the recurrences, equivalences and termination of wfa_kernels.cu (see its
// header): scores visited in steps of g = gcd(x, o, e), only the diagonals
// the sources reach, intersected with the reference's [lo, hi] (:158-164),
// negative values stored as NEG.
//
// Storage.  A pair's M/I/D rings (nslot = hm + 2*hie slots, 9 for x4 o6 e2)
// live in a window of W int16 elements per slot, diagonal k at element
// H + k.  The visited interval after S steps lies inside [-S, S] (a source
// reaches one diagonal further per step), so the window fills from its
// centre outwards and every element is NEG-filled once when the pair starts;
// afterwards each step only overwrites its own interval and turns what the
// reused slot held outside it back into NEG where a later step could read it.
// Reads at k-1 and k+1 therefore need no bounds tests.
//
// A step.  A thread takes groups of four (or, for the last round, two)
// neighbouring diagonals: rows come in as 8-byte loads, the recurrences are
// 16-bit-pair DPX on two diagonals per register, and only the extension is per
// diagonal (wf_group).  The intervals are packed (lo, -hi) pairs, so that unions,
// widening and clipping are single DPX instructions too.  Before, every thread took
// single diagonals TW apart: 20,000 pairs of 100-10,000 bp went from 16.5 to 11.9 ms,
// of which the groups 16.5 -> 13.9 (with the packed intervals), the sequence copies
// below 13.9 -> 12.4, one inlined extension loop for a lane's diagonals 12.4 -> 12.1.
//
// Tiers.  Work per pair grows with the square of its cost (most pairs are
// cheap, most cells are in the few expensive ones), so a pair starts on a
// small team and moves up when its interval outgrows the window:
//   T1   one warp per pair,      sixteen per block, W = 632  (x4 o6 e2)
//   T2   two warps per pair,     eight per block,   W = 1,264
//   T4   four warps per pair,    four per block,    W = 2,760
//   T8   eight warps per pair,   two per block,     W = 5,536
//   T16  sixteen warps per pair, one per block,     W = 11,976
// each in its own launch, one after another on the executor's stream.  A
// pair whose next step would read or write outside its window is suspended:
// the team writes its state (step intervals, step, ring contents over the
// live span) to a dump record in HBM and queues the pair for the next tier,
// whose launch restores it into its larger window and continues from the
// same step.  No cell is computed twice.  A pair that outgrows T16, or whose
// rows could leave int16 (qlen + steps > 32767), runs from the start in the
// G tier: sixteen warps per pair with int32 rings in a per-block region of
// global memory large enough for any interval ([-max(qlen, rlen) - 3, ...]).
// When the dump space of a transition is used up, the pair starts over in
// the next tier instead (same results, more work).
//
// Sequences are copied into shared memory as 16-base words, so a 16-base window at
// any position is two neighbouring words and one funnel shift; pairs longer than a
// tier's copy capacity read their windows from the packed words in global memory.
//
// Bound: instruction issue: 77 thread instructions per cell, most of them the extension's
// two window loads, shifts, compare and clamps and a step's bookkeeping.  20,000 pairs of
// 100-10,000 bp (2.7e9 cells, by counters): T1 2.5 ms at 71% of the issue slots, the bound
// pass 2.0 at 64%, T4 5.9 at 63%, sixteen warps per SM each.
#include <algorithm>
#include <type_traits>

#include "gb2_internal.cuh"

namespace gb2 {
namespace {

constexpr int32_t kPromote = -10;  // suspended: the pair continues in the next tier
constexpr int32_t kRestart = -11;  // must start over in the G tier (int32 rings)
constexpr int32_t kRunning = -12;  // internal: no result yet
constexpr int kDumpHeader = 1024;  // bytes of a dump record before the ring data

struct Shape {
    int g, xs, oes, es, hm, hie, nslot;
};

__device__ __forceinline__ int gcd_d(int a, int b)
{
    while (b) {
        const int t = a % b;
        a = b;
        b = t;
    }
    return a;
}

__device__ __forceinline__ Shape make_shape(const WfaParams &p)
{
    Shape w;
    w.g = gcd_d(p.x, gcd_d(p.o, p.e));
    w.xs = p.x / w.g;
    w.oes = (p.o + p.e) / w.g;
    w.es = p.e / w.g;
    w.hm = max(w.xs, w.oes) + 1;
    w.hie = w.es + 1;
    w.nslot = w.hm + 2 * w.hie;
    return w;
}

// ---- team synchronisation ----------------------------------------------------
// TEAM warps align one pair; a block holds NTEAMS teams.  A whole block uses
// __syncthreads, a part of a block a named barrier (id 1 + team), a warp
// __syncwarp.  Both forms order shared and global memory among the team.
template <int TEAM, int NTEAMS>
struct Team {
    int id;  // team index in the block
    __device__ __forceinline__ void sync() const
    {
        if (TEAM == 1)
            __syncwarp();
        else if (NTEAMS == 1)
            __syncthreads();
        else
            asm volatile("bar.sync %0, %1;" ::"r"(1 + id), "r"(TEAM * 32) : "memory");
    }
    // barrier that also ORs v over the team
    __device__ __forceinline__ bool any(bool v) const
    {
        if (TEAM == 1) {
            __syncwarp();
            return __any_sync(0xffffffffu, v);
        }
        if (NTEAMS == 1)
            return __syncthreads_or(v) != 0;
        uint32_t res;
        asm volatile(
            "{\n\t.reg .pred pi, po;\n\t"
            "setp.ne.u32 pi, %1, 0;\n\t"
            "bar.red.or.pred po, %2, %3, pi;\n\t"
            "selp.u32 %0, 1, 0, po;\n\t}"
            : "=r"(res)
            : "r"((uint32_t)v), "r"(1 + id), "r"(TEAM * 32)
            : "memory");
        return res != 0;
    }
};

// ---- sequences ---------------------------------------------------------------
// 16-base windows of a sequence: from the shared copy (16-base words in order, first
// base on top) or from the packed little-endian words in global memory (logical word j
// at 32-bit index j ^ 1, clamped to the array).
struct SeqWin {
    const uint32_t *win;
    const uint32_t *w32;
    int32_t last;
};

template <bool SMEM>
__device__ __forceinline__ uint32_t win16(const SeqWin &s, int32_t pos)
{
    const int32_t j = pos >> 4;
    if (SMEM)
        return __funnelshift_l(s.win[j + 1], s.win[j], (uint32_t)pos << 1);
    const uint32_t hi = __ldg(s.w32 + ((uint32_t)j ^ 1u));
    const uint32_t lo = __ldg(s.w32 + ((uint32_t)min(j + 1, s.last) ^ 1u));
    return __funnelshift_l(lo, hi, (uint32_t)pos << 1);
}

// Bytes that must be readable past the last copy of a block (ext_more).
constexpr int32_t kSeqSlack = 16;

// Copies nw packed words into win[0 .. 2*nw) when SMEM, and two guard words after them,
// whose bases match nothing in the other sequence's guard.  (One word per 16 bases and
// two loads per window, instead of overlapping 64-bit windows and one: the one-warp
// tier's copy holds 6,144 bases in 3 KB, where it held 2,048 in 2 KB and longer pairs
// read their windows from global memory.)
template <bool SMEM>
__device__ __forceinline__ SeqWin stage_seq(const SeqView &v, int64_t off, int32_t nw,
                                            uint32_t *win, int tt, int tw, uint32_t guard)
{
    if (SMEM) {
        const uint64_t *src = v.packed + off;
        for (int32_t i = tt; i < nw; i += tw) {
            const uint64_t a = __ldg(src + i);
            *reinterpret_cast<uint2 *>(win + 2 * i) =
                make_uint2((uint32_t)(a >> 32), (uint32_t)a);
        }
        if (tt == 0)
            *reinterpret_cast<uint2 *>(win + 2 * nw) = make_uint2(guard, guard);
        return SeqWin{win, nullptr, 0};
    }
    const int64_t last = 2 * (v.n_words - off) - 1;
    return SeqWin{nullptr, reinterpret_cast<const uint32_t *>(v.packed + off),
                  (int32_t)min(last, (int64_t)0x7fffffff)};
}

// Extend along diagonal k from row (align_cpu.mojo:208-219): XOR of the two
// 16-base windows, leading zeros / 2 = matching bases, clamped by the
// remaining lengths.  Requires row >= 0 and row - k >= 0.
template <bool SMEM>
__device__ __forceinline__ int32_t ext_more(const SeqWin &qs, int32_t qlen, const SeqWin &rs,
                                           int32_t rlen, int32_t row, int32_t k)
{
    const int32_t end = min(qlen, rlen + k);
    while (row < end) {
        // four windows at once: their loads do not wait for one another
        uint32_t x[4];
        if (SMEM) {
            // five neighbouring words of each copy; those past its end (the four words
            // kSeqSlack leaves readable) only match past `end`
            const uint32_t *const a = qs.win + (row >> 4), *const b = rs.win + ((row - k) >> 4);
            const uint32_t sa = (uint32_t)row << 1, sb = (uint32_t)(row - k) << 1;
            uint32_t wa = a[0], wb = b[0];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t na = a[i + 1], nb = b[i + 1];
                x[i] = __funnelshift_l(na, wa, sa) ^ __funnelshift_l(nb, wb, sb);
                wa = na;
                wb = nb;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int32_t at = min(row + 16 * i, end - 1);
                x[i] = win16<false>(qs, at) ^ win16<false>(rs, at - k);
            }
        }
        const uint32_t y = x[0] ? x[0] : x[1] ? x[1] : x[2] ? x[2] : x[3];
        row += (x[0] ? 0 : x[1] ? 16 : x[2] ? 32 : 48) + (__clz((int)y) >> 1);
        if (y)
            break;
    }
    return min(row, end);
}

template <bool SMEM>
__device__ __noinline__ int32_t ext_run(const SeqWin &qs, int32_t qlen, const SeqWin &rs,
                                        int32_t rlen, int32_t row, int32_t k)
{
    return ext_more<SMEM>(qs, qlen, rs, rlen, row, k);
}

// First window of U diagonals at once; the ones whose whole window matched
// go on one by one.  In range: 0 <= row < qlen and 0 <= row - k < rlen.
template <int U, bool SMEM>
__device__ __forceinline__ void ext_u(const SeqWin &qs, int32_t qlen, const SeqWin &rs,
                                      int32_t rlen, int32_t (&rows)[U], const int32_t (&ks)[U],
                                      const bool (&live)[U])
{
    // Either sequence empty: no diagonal can extend (and there is no window to load).
    if (qlen <= 0 || rlen <= 0)
        return;
    // Live rows are >= 0 (and so are their columns); dead rows are negative and
    // must not move.  Window positions are clamped into the sequences, so every
    // load is in bounds, and the advance max(0, min(ml, qlen - row, rlen - col))
    // is zeroed for dead rows and for diagonals past the last one.
    int32_t adv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int32_t row = rows[u], col = row - ks[u];
        const int32_t pq = (int32_t)min((uint32_t)row, (uint32_t)(qlen - 1));
        const int32_t pr = (int32_t)min((uint32_t)col, (uint32_t)(rlen - 1));
        const uint32_t x = win16<SMEM>(qs, pq) ^ win16<SMEM>(rs, pr);
        int32_t ml = __clz((int)x) >> 1;
        ml += ml >> 4;  // 17 for a whole matching window
        int32_t a = __vimin3_s32_relu(ml, qlen - row, rlen - col);
        a &= ~(row >> 31);
        if (!live[u])
            a = 0;
        adv[u] = a;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        // 17: the window matched and both sequences go on past it: the rest one by one
        if (adv[u] == 17)
            rows[u] = ext_run<SMEM>(qs, qlen, rs, rlen, rows[u] + 16, ks[u]);
        else
            rows[u] += adv[u];
    }
}

// N = 4 or 2 neighbouring diagonals of one step in int16 rings: window positions p0 ..
// p0 + N - 1 (p0 a multiple of N), diagonals k0 on; positions outside [pa, pb] are stored
// as NEG.  Rows point at window position 0.  Two diagonals per register: the rows come in
// by N-element loads and 4-byte ones for the neighbours left and right (N = 4: 8 loads and
// 7 permutes for what were 20 two-byte loads), and the recurrences are 16-bit-pair DPX.
// The extension is per diagonal: positions are kept doubled (bit offsets into the packed
// bases), clamped unsigned so that a dead row -- negative, and so is its column -- reads
// the two guard windows, which differ in their first base: it advances by 0 without a
// test.
template <int N, bool SMEM>
__device__ __forceinline__ void wf_group(const int16_t *Mx, const int16_t *Moe, const int16_t *Ie,
                                         const int16_t *De, int16_t *Mw, int16_t *Iw, int16_t *Dw,
                                         int32_t p0, int32_t k0, int32_t pa, int32_t pb,
                                         const SeqWin &qs, int32_t qlen, const SeqWin &rs,
                                         int32_t rlen, uint32_t qguard2, uint32_t rguard2)
{
    constexpr int P = N / 2;  // registers of two diagonals
    const uint32_t NEG2 = 0x80008000u, ONE2 = 0x00010001u;
    auto load = [&](const int16_t *row, uint32_t (&v)[P]) {
        if (N == 4) {
            const uint2 t = *reinterpret_cast<const uint2 *>(row + p0);
            v[0] = t.x;
            v[P - 1] = t.y;
        } else {
            v[0] = *reinterpret_cast<const uint32_t *>(row + p0);
        }
    };
    auto store = [&](int16_t *row, const uint32_t (&v)[P]) {
        if (N == 4)
            *reinterpret_cast<uint2 *>(row + p0) = make_uint2(v[0], v[P - 1]);
        else
            *reinterpret_cast<uint32_t *>(row + p0) = v[0];
    };
    auto pair_at = [&](const int16_t *row, int off) {
        return *reinterpret_cast<const uint32_t *>(row + p0 + off);
    };
    uint32_t mx[P], mo[P], ie[P], de[P];
    load(Mx, mx);
    load(Moe, mo);
    load(Ie, ie);
    load(De, de);
    const uint32_t mol = pair_at(Moe, -2), mor = pair_at(Moe, N), iel = pair_at(Ie, -2),
                   der = pair_at(De, N);
    uint32_t iv[P], dv[P], mv[P];
#pragma unroll
    for (int j = 0; j < P; ++j) {
        // elements k - 1 of M and I, k + 1 of M and D, for the two diagonals k
        const uint32_t ml = __byte_perm(j ? mo[j ? j - 1 : 0] : mol, mo[j], 0x5432);
        const uint32_t il = __byte_perm(j ? ie[j ? j - 1 : 0] : iel, ie[j], 0x5432);
        const uint32_t mr = __byte_perm(mo[j], j + 1 < P ? mo[j + 1 < P ? j + 1 : j] : mor, 0x5432);
        const uint32_t dr = __byte_perm(de[j], j + 1 < P ? de[j + 1 < P ? j + 1 : j] : der, 0x5432);
        const uint32_t i0 = __vmaxs2(ml, il);
        dv[j] = __vmaxs2(mr, dr);
        // max(mx + 1, i + 1, d)
        mv[j] = __viaddmax_s16x2(mx[j], ONE2, __viaddmax_s16x2(i0, ONE2, dv[j]));
        iv[j] = __viaddmax_s16x2(i0, ONE2, NEG2);
    }
    if (qlen > 0 && rlen > 0) {
        int32_t row[N], end[N];
        uint32_t x[N];
        uint32_t least = 0xFFFFFFFFu;
#pragma unroll
        for (int u = 0; u < N; ++u) {
            row[u] = (u & 1) ? (int32_t)mv[u / 2] >> 16 : (int32_t)(int16_t)mv[u / 2];
            end[u] = __viaddmin_s32(k0 + u, rlen, qlen);  // last row of the diagonal
            if (SMEM) {
                const uint32_t q2 = __viaddmin_u32((uint32_t)row[u], (uint32_t)row[u], qguard2);
                const uint32_t r2 = __viaddmin_u32(2u * (uint32_t)row[u],
                                                   (uint32_t)(-2 * (k0 + u)), rguard2);
                const uint32_t *const a = reinterpret_cast<const uint32_t *>(
                    reinterpret_cast<const char *>(qs.win) + ((q2 >> 3) & ~3u));
                const uint32_t *const b = reinterpret_cast<const uint32_t *>(
                    reinterpret_cast<const char *>(rs.win) + ((r2 >> 3) & ~3u));
                x[u] = __funnelshift_l(a[1], a[0], q2) ^ __funnelshift_l(b[1], b[0], r2);
            } else {
                const int32_t pq = (int32_t)min((uint32_t)row[u], (uint32_t)(qlen - 1));
                const int32_t pr = (int32_t)min((uint32_t)(row[u] - k0 - u), (uint32_t)(rlen - 1));
                x[u] = row[u] < 0 ? 0xFFFFFFFFu : win16<false>(qs, pq) ^ win16<false>(rs, pr);
            }
            least = min(least, x[u]);
        }
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const int32_t adv = __clz((int)x[u]) >> 1;  // 16 for a whole matching window
            row[u] = max(row[u], __viaddmin_s32(row[u], adv, end[u]));
        }
        // whole windows matched: those diagonals go on by themselves, the lanes' together
        if (least == 0) {
            uint32_t todo = 0;
#pragma unroll
            for (int u = 0; u < N; ++u)
                todo |= x[u] == 0 && row[u] < end[u] ? 1u << u : 0u;
            while (todo) {
                const int v = __ffs((int)todo) - 1;
                todo &= todo - 1;
                int32_t at = row[0];
#pragma unroll
                for (int u = 1; u < N; ++u)
                    at = v == u ? row[u] : at;
                at = ext_more<SMEM>(qs, qlen, rs, rlen, at, k0 + v);
#pragma unroll
                for (int u = 0; u < N; ++u)
                    row[u] = v == u ? at : row[u];
            }
        }
#pragma unroll
        for (int j = 0; j < P; ++j)
            mv[j] = __byte_perm((uint32_t)row[2 * j], (uint32_t)row[2 * j + 1], 0x5410);
    }
    if (p0 < pa || p0 + N - 1 > pb) {  // the interval's ends
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const int32_t e0 = p0 + 2 * j, e1 = e0 + 1;
            const uint32_t keep = (e0 >= pa && e0 <= pb ? 0xFFFFu : 0u) |
                                  (e1 >= pa && e1 <= pb ? 0xFFFF0000u : 0u);
            mv[j] = (mv[j] & keep) | (NEG2 & ~keep);
            iv[j] = (iv[j] & keep) | (NEG2 & ~keep);
            dv[j] = (dv[j] & keep) | (NEG2 & ~keep);
        }
    }
    store(Iw, iv);
    store(Dw, dv);
    store(Mw, mv);
}

// ---- dump records ---------------------------------------------------------------
// A suspended pair: int32 header {next step, M slot, I/D slot, span lo, span
// hi} at 0, {lo, hi} of the step in M slot j at int 32 + 2j, and
// from byte kDumpHeader the nslot ring rows over [span lo, span hi], each
// span elements of int16.
//
// The shared-memory tiers write the rows with one bulk asynchronous copy per
// row (cp.async.bulk from this CTA's shared memory to global), which needs both
// addresses and the size in whole 16-byte units.  So the span is the live
// span widened outward to diagonals whose window positions H + k are
// multiples of 8: the window's rows start on 16 bytes (W is a multiple of 8,
// the ring 16-byte aligned) and hold positions [0, W), so the widened span
// stays inside the row; outside every slot's interval a row holds NEG, so the
// extra elements are NEG.  Records lie whole multiples of 256 bytes apart and
// the rows at kDumpHeader + j * span * 2 with span a multiple of 8; the
// alignment is checked when a record is written (an element copy otherwise).
// The larger window a record is restored into holds the widened span too (its
// H and W - H are no smaller), where the extra NEGs land on NEG.
__device__ __forceinline__ void bulk_row_to_global(void *dst, const void *src_smem,
                                                   uint32_t bytes)
{
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(src_smem);
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                 :: "l"(dst), "r"(s), "r"(bytes) : "memory");
}
struct DumpOut {
    uint8_t *base;      // records of dump_stride bytes
    int64_t stride;
    int64_t cap;        // records available
    int *ctr;           // records claimed
};

// ---- one pair, int16 rings ------------------------------------------------------
// Aligns pair pi with this team.  ring: the team's window (nslot rows of W elements,
// diagonal k of slot j at ring[j * W + H + k]).  resume: a dump record to continue
// from, or nullptr.  Returns the cost (>= 0), -1 past max_error, kPromote (state
// written to record *dump_idx, or *dump_idx = -1 when no record was free), or kRestart
// (int16 rows would overflow).  The return value is uniform over the team.
//
// Intervals.  A step's diagonals [lo, hi] are kept as (lo, -hi) in the halves of one
// register, kNone when there are none, so that the union of sources is a 16-bit-pair
// minimum, one diagonal further a -1 in both halves, and clipping a maximum.  Lane j
// holds those of the step in M slot j: of its M (ivm) and of its I and D (ivi), which
// start later (no step reached by mismatches alone has any).  Diagonals of a window
// fit 14 bits; limits beyond it are cut to +-kFar.
constexpr uint32_t kNone = 0x3FFF3FFFu;
constexpr int32_t kFar = 16000;

__device__ __forceinline__ uint32_t pack2(int32_t lo, int32_t nhi)
{
    return __byte_perm((uint32_t)lo, (uint32_t)nhi, 0x5410);
}
__device__ __forceinline__ int32_t cut(int32_t v) { return min(max(v, -kFar), kFar); }

template <int TEAM, int NTEAMS, bool SMEM_SEQ>
__device__ __forceinline__ int32_t tier_pair16(
    const SeqView &q, const SeqView &r, const WfaParams &p, const Shape &w, int64_t pi,
    int16_t *ring, int32_t W, int32_t H, uint32_t *sq, uint32_t *sr, const Team<TEAM, NTEAMS> &team,
    volatile int64_t *bcast, const uint8_t *resume, const DumpOut &dump, int64_t *dump_idx,
    int64_t &cells, int32_t band_w, int32_t ub)
{
    constexpr int TW = TEAM * 32;
    const unsigned FULL = 0xffffffffu;
    const uint32_t ONES = 0xFFFFFFFFu;  // -1 in both halves
    const int lane = threadIdx.x & 31;
    const int tt = (int)(threadIdx.x % TW);
    const int hm = w.hm, hie = w.hie, xs = w.xs, oes = w.oes, es = w.es, g = w.g;
    const int32_t max_err = p.max_error;
    const int64_t qoff = q.offsets[pi] - q.word_base;
    const int64_t roff = r.offsets[pi] - r.word_base;
    const int32_t qlen = (int32_t)q.lengths[pi], rlen = (int32_t)r.lengths[pi];
    if (qlen == 0 && rlen == 0)
        return 0;
    const int32_t qnw = (qlen + 31) >> 5, rnw = (rlen + 31) >> 5;
    team.sync();  // the previous pair's reads of the shared copies and the ring are done
    const SeqWin qs = stage_seq<SMEM_SEQ>(q, qoff, qnw, sq, tt, TW, 0u);
    const SeqWin rs = stage_seq<SMEM_SEQ>(r, roff, rnw, sr, tt, TW, 0xFFFFFFFFu);
    {
        // every ring element NEG (W is a multiple of 8 and the window 16-byte aligned)
        uint4 *v = reinterpret_cast<uint4 *>(ring);
        const uint4 n4 = make_uint4(0x80008000u, 0x80008000u, 0x80008000u, 0x80008000u);
        for (int32_t i = tt; i < w.nslot * W / 8; i += TW)
            v[i] = n4;
    }
    const int32_t target = qlen - rlen;
    // doubled positions of the guard windows
    const uint32_t qguard2 = (uint32_t)qnw * 64u, rguard2 = (uint32_t)rnw * 64u;
    uint32_t ivm = kNone, ivi = kNone;
    int ms = 0, is = 0;
    int32_t sp = 1;
    team.sync();  // NEG fill done before the restored / initial values land
    if (resume) {
        const int32_t *hd = reinterpret_cast<const int32_t *>(resume);
        sp = hd[0];
        ms = hd[1];
        is = hd[2];
        const int32_t ulo = hd[3], uhi = hd[4];
        ivm = (uint32_t)hd[32 + 2 * lane];
        ivi = (uint32_t)hd[33 + 2 * lane];
        const int32_t span = uhi - ulo + 1;
        if (span > 0) {
            const int16_t *src = reinterpret_cast<const int16_t *>(resume + kDumpHeader);
            const int32_t total = w.nslot * span;
            for (int32_t i = tt; i < total; i += TW) {
                const int32_t j = i / span, kk = i - j * span;
                ring[j * W + H + ulo + kk] = src[i];
            }
        }
    } else {
        // score 0: M[0,0] = 0 extended along diagonal 0 (:130-140)
        const int32_t row0 = ext_run<SMEM_SEQ>(qs, qlen, rs, rlen, 0, 0);
        if (lane == 0)
            ivm = 0;
        if (tt == 0)
            ring[H] = (int16_t)row0;
        cells += 1;
        if (target == 0 && row0 >= qlen)
            return 0;
    }
    team.sync();
    // limits that do not change: the matrix, then [target] let in, then max_error and
    // the bound pass's band (around the line from diagonal 0 to the target)
    const int32_t tc = cut(target);
    const uint32_t lim_matrix = pack2(-min(rlen, kFar), -min(qlen, kFar));
    const uint32_t lim_target = pack2(tc, -tc);
    // (through a shuffle: where maxima met a negated kernel argument, a build with CUDA 12.9
    // was seen to clip at +max_err)
    int32_t flo = __shfl_sync(FULL, -min(max_err, kFar), 0), fnhi = flo;
    if (band_w > 0) {
        flo = max(flo, cut(min(0, target) - band_w));
        fnhi = max(fnhi, cut(-max(0, target) - band_w));
    }
    const uint32_t lim_fixed = pack2(flo, fnhi);
    // a step reads whole groups of four and the pairs beside them
    const uint32_t lim_window = pack2(4 - H, -(W - 6 - H));
    // pruning by the upper bound ub: R = (ub - s) / e at the next step, kept as quotient
    // and remainder; the diagonals [target - R, target + R]
    int32_t plo = -(1 << 30), pnhi = -(1 << 30), rr = 0;
    if (ub >= 0) {
        const int32_t num = ub - sp * g, rq = num / p.e;
        rr = num - rq * p.e;
        plo = target - rq;
        pnhi = -target - rq;
    }
    // row offsets, in elements: the step's own rows and its sources'.  A source before
    // the first step falls on a slot not written yet, which is NEG with no interval.
    const int32_t mrows = hm * W, irows = hie * W;
    int32_t om = ms * W, oi = is * W;
    // steps s = sp * g <= max_err; int16 rows are proven for sp <= 32767 - qlen, and a dead
    // row (NEG plus at most one per step) has a negative column on every diagonal of the
    // window while sp < 32768 - H
    const int32_t sp_end = max_err / g;
    const int32_t sp_lim = min(sp_end, 32767 - max(qlen, H + 8));
    for (; sp <= sp_lim; ++sp) {
        const int32_t s = sp * g;
        const int nms = ms + 1 == hm ? 0 : ms + 1;
        const int sx = nms >= xs ? nms - xs : nms - xs + hm;
        const int soe = nms >= oes ? nms - oes : nms - oes + hm;
        const int se = nms >= es ? nms - es : nms - es + hm;
        const uint32_t vx = __shfl_sync(FULL, ivm, sx);
        const uint32_t voe = __shfl_sync(FULL, ivm, soe);
        const uint32_t ve = __shfl_sync(FULL, ivi, se);
        // I and D: the sources one diagonal further out (kNone stays above every limit)
        const uint32_t vid = __viaddmax_s16x2(__vmins2(voe, ve), ONES, 0x80008000u);
        const uint32_t vall = __vmins2(vid, vx);
        uint32_t lim = __vmaxs2(lim_matrix, pack2(-min(s, kFar), -min(s, kFar)));
        lim = __vmaxs2(__vmins2(lim, lim_target), lim_fixed);
        if (ub >= 0) {
            // a diagonal k at score s costs at least s + e*|k - target| to finish (every
            // diagonal change is a gap base): beyond the upper bound ub it cannot be on an
            // alignment of cost <= ub, and dropping it only lowers values elsewhere, so the
            // first hit stays at the same s
            lim = __vmaxs2(lim, pack2(cut(plo), cut(pnhi)));
            rr -= g;
            if (rr < 0) {
                rr += p.e;
                ++plo;
                ++pnhi;
            }
        }
        const uint32_t ab = __vmaxs2(vall, lim);
        const int32_t a = (int32_t)(int16_t)ab, b = -((int32_t)ab >> 16);
        const bool empty = a > b;
        if (!empty && __vmaxs2(ab, lim_window) != ab) {
            // outside the window: the pair moves to the next tier, in the state after
            // step sp - 1
            int64_t di = -1;
            if (dump.base) {
                if (tt == 0) {
                    const int64_t c = atomicAdd(dump.ctr, 1);
                    *bcast = c < dump.cap ? c : -1;
                }
                team.sync();
                di = *bcast;
                team.sync();  // read by every thread before the slot is reused
            }
            if (di >= 0) {
                uint8_t *rec = dump.base + di * dump.stride;
                int32_t *hd = reinterpret_cast<int32_t *>(rec);
                // the live span: the union of every step's interval, widened to 16-byte
                // units of the window rows
                const int32_t l = (int32_t)(int16_t)ivm, nh = (int32_t)ivm >> 16;
                const bool some = lane < hm && l + nh <= 0;
                int32_t l0 = __reduce_min_sync(FULL, some ? l : 0x7fffffff);
                int32_t h0 = __reduce_max_sync(FULL, some ? -nh : -0x7fffffff);
                if (l0 <= h0) {
                    l0 -= (H + l0) & 7;
                    h0 += 7 - ((H + h0) & 7);
                }
                if (tt == 0) {
                    hd[0] = sp;
                    hd[1] = ms;
                    hd[2] = is;
                    hd[3] = l0;
                    hd[4] = h0;
                }
                if (tt < 32) {
                    hd[32 + 2 * lane] = (int32_t)ivm;
                    hd[33 + 2 * lane] = (int32_t)ivi;
                }
                const int32_t span = h0 - l0 + 1;
                if (span > 0) {
                    int16_t *dst = reinterpret_cast<int16_t *>(rec + kDumpHeader);
                    // alignment as derived above, checked (the same on every thread of
                    // the team): the element copy below otherwise
                    const bool bulk = (((uintptr_t)dst & 15u) == 0) && ((W & 7) == 0) &&
                                      ((__cvta_generic_to_shared(ring + H + l0) & 15u) == 0);
                    if (bulk) {
                        // every thread orders its ring writes before the async proxy's
                        // reads, then one thread hands the rows to the copy engine and
                        // waits for them before the team can reuse the window (the next
                        // pair starts with a barrier)
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        team.sync();
                        if (tt == 0) {
                            for (int j = 0; j < w.nslot; ++j)
                                bulk_row_to_global(dst + (int64_t)j * span, ring + j * W + H + l0,
                                                   (uint32_t)span * 2u);
                            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
                        }
                    } else {
                        const int32_t total = w.nslot * span;
                        for (int32_t i = tt; i < total; i += TW) {
                            const int32_t j = i / span, kk = i - j * span;
                            dst[i] = ring[j * W + H + l0 + kk];
                        }
                    }
                }
            }
            *dump_idx = di;
            return kPromote;
        }
        ms = nms;
        is = is + 1 == hie ? 0 : is + 1;
        om = om + W == mrows ? 0 : om + W;
        oi = oi + W == irows ? 0 : oi + W;
        // What the reused slots held (the steps sp - hm for M, sp - hie for I and D) and
        // this step does not overwrite becomes NEG.  Not on a side that the pruning bound
        // cuts (ab above vall): the bound closes in by one diagonal per e of score, so a
        // later step that reads this slot -- at e or o + e more, one diagonal further out,
        // or at x more on the same diagonals -- stays inside [a, b] on that side.
        const uint32_t old = __vmins2(__shfl_sync(FULL, ivm, ms),
                                      __shfl_sync(FULL, ivi, ms >= hie ? ms - hie : ms - hie + hm));
        int16_t *const Mw = ring + om, *const Iw = ring + mrows + oi, *const Dw = Iw + irows;
        if (empty || __vmins2(old, ab) != ab) {
            const int32_t olo = (int32_t)(int16_t)old, ohi = -((int32_t)old >> 16);
            const uint32_t cutd = ab ^ vall;
            // an unclipped side is cleaned up to the interval's end
            const int32_t le = empty ? ohi : ((cutd & 0xFFFFu) ? olo - 1 : min(ohi, a - 1));
            const int32_t rs0 = empty ? ohi + 1 : ((cutd >> 16) ? ohi + 1 : max(olo, b + 1));
            if (olo <= ohi) {
                for (int32_t k = olo + tt; k <= le; k += TW)
                    Mw[H + k] = Iw[H + k] = Dw[H + k] = (int16_t)-32768;
                for (int32_t k = rs0 + tt; k <= ohi; k += TW)
                    Mw[H + k] = Iw[H + k] = Dw[H + k] = (int16_t)-32768;
            }  // where the groups below reach over these, they write NEG too
        }
        if (!empty) {
            cells += (int64_t)(b - a + 1);
            const int16_t *const Mx = ring + sx * W, *const Moe = ring + soe * W;
            const int16_t *const Ie = ring + mrows + (oi >= es * W ? oi - es * W
                                                                   : oi - es * W + irows);
            const int16_t *const De = Ie + irows;
            const int32_t pa = H + a, pb = H + b;
            // groups of neighbouring diagonals, one per thread and round: of four while
            // more are left than a round of two covers, which wastes fewer threads on
            // the last one
            int32_t p0 = pa & ~3;
            for (; pb - p0 >= 2 * TW; p0 += 4 * TW) {
                const int32_t at = p0 + 4 * tt;
                if (at <= pb)
                    wf_group<4, SMEM_SEQ>(Mx, Moe, Ie, De, Mw, Iw, Dw, at, at - H, pa, pb, qs,
                                          qlen, rs, rlen, qguard2, rguard2);
            }
            p0 += 2 * tt;
            if (p0 <= pb)
                wf_group<2, SMEM_SEQ>(Mx, Moe, Ie, De, Mw, Iw, Dw, p0, p0 - H, pa, pb, qs, qlen,
                                      rs, rlen, qguard2, rguard2);
        }
        if (lane == ms) {
            ivm = empty ? kNone : ab;
            // I and D cover the step's diagonals, but no more than their own sources reach
            const uint32_t own = __vmaxs2(vid, lim);
            ivi = empty || (int32_t)(int16_t)own + ((int32_t)own >> 16) > 0 ? kNone : own;
        }
        team.sync();
        // M[s, target] >= qlen ends the alignment (:221-224)
        if (a <= target && target <= b && (int32_t)Mw[H + target] >= qlen)
            return s;
    }
    return sp <= sp_end ? kRestart  // past the steps int16 values are proven for
                        : -1;       // the loop ran out: cost above max_error (:226)
}

// ---- one pair, int32 rings (the G tier) ---------------------------------------------
// As above over int32 rings in global memory that hold every diagonal: pairs start over
// here, never move on, and write one diagonal per thread and round.
template <int TEAM, int NTEAMS, int U, bool SMEM_SEQ>
__device__ __forceinline__ int32_t tier_pair32(const SeqView &q, const SeqView &r,
                                               const WfaParams &p, const Shape &w, int64_t pi,
                                               int32_t *ring, int32_t W, int32_t H, uint32_t *sq,
                                               uint32_t *sr, const Team<TEAM, NTEAMS> &team,
                                               int64_t &cells, int32_t ub)
{
    constexpr int TW = TEAM * 32;
    using RT = int32_t;
    constexpr int32_t NEG = -(1 << 30);
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int tt = (int)(threadIdx.x % TW);
    const int hm = w.hm, hie = w.hie, xs = w.xs, oes = w.oes, es = w.es, g = w.g;
    const int32_t max_err = p.max_error;
    const int32_t neg_err = __shfl_sync(FULL, -max_err, 0);  // see flo above
    const int64_t qoff = q.offsets[pi] - q.word_base;
    const int64_t roff = r.offsets[pi] - r.word_base;
    const int32_t qlen = (int32_t)q.lengths[pi], rlen = (int32_t)r.lengths[pi];
    if (qlen == 0 && rlen == 0)
        return 0;
    const int32_t qnw = (qlen + 31) >> 5, rnw = (rlen + 31) >> 5;
    team.sync();  // the previous pair's reads of the shared copies and the ring are done
    const SeqWin qs = stage_seq<SMEM_SEQ>(q, qoff, qnw, sq, tt, TW, 0u);
    const SeqWin rs = stage_seq<SMEM_SEQ>(r, roff, rnw, sr, tt, TW, 0xFFFFFFFFu);
    // the slots and the NEG row; more than 2^31 elements for sequences of some 10^8 bases
    for (int64_t i = tt; i < (int64_t)(w.nslot + 1) * W; i += TW)
        ring[i] = NEG;
    const int32_t target = qlen - rlen;
    RT *const base = ring + H;
    auto slot = [&](int j) { return base + (int64_t)j * W; };
    // per-slot intervals: lane j holds M slot j's and I/D slot j's
    int32_t mlo = 1, mhi = 0, ilo = 1, ihi = 0;
    int ms = 0, is = 0;
    const int64_t sp0 = 1;
    int32_t result = kRunning;
    team.sync();  // NEG fill done before the restored / initial values land
    {
        // score 0: M[0,0] = 0 extended along diagonal 0 (:130-140)
        const int32_t row0 = ext_run<SMEM_SEQ>(qs, qlen, rs, rlen, 0, 0);
        if (lane == 0) {
            mlo = 0;
            mhi = 0;
        }
        if (tt == 0)
            slot(0)[0] = (RT)row0;
        cells += 1;
        if (target == 0 && row0 >= qlen)
            result = 0;
    }
    team.sync();
    int32_t rq = 0, rr = 0;  // pruning: (ub - s) / e and its remainder at s = sp0 * g
    if (ub >= 0) {
        const int32_t num = ub - (int32_t)(sp0 * g);
        rq = num / p.e;
        rr = num - rq * p.e;
    }
    if (result == kRunning) {
        const int32_t sp_end = max_err / g;  // steps s = sp * g <= max_err
        int32_t sp = (int32_t)sp0;
        for (; sp <= sp_end; ++sp) {
            const int32_t s = (int32_t)(sp * g);
            const int nms = ms + 1 == hm ? 0 : ms + 1;
            const int nis = is + 1 == hie ? 0 : is + 1;
            int32_t lo = max(-rlen, -s), hi = min(qlen, s);
            if (target < lo || target > hi) {
                lo = min(lo, target);
                hi = max(hi, target);
            }
            lo = max(lo, neg_err);
            hi = min(hi, max_err);
            if (ub >= 0) {
                // a diagonal k at score s costs at least s + e*|k - target| to finish
                // (every diagonal change is a gap base): beyond the upper bound ub it
                // cannot be on an alignment of cost <= ub, and dropping it only
                // lowers values elsewhere, so the first hit stays at the same s
                // R = (ub - s) / e, kept as quotient and remainder (s grows by g
                // per step, and ub >= s while the pair runs)
                const int32_t R = rq;
                rr -= g;
                if (rr < 0) {
                    rr += p.e;
                    --rq;
                }
                lo = max(lo, target - R);
                hi = min(hi, target + R);
            }
            const int sx = sp >= xs ? (nms >= xs ? nms - xs : nms - xs + hm) : -1;
            const int soe = sp >= oes ? (nms >= oes ? nms - oes : nms - oes + hm) : -1;
            const int se = sp >= es ? (nis >= es ? nis - es : nis - es + hie) : -1;
            int32_t ulo = 0x7fffffff, uhi = -0x7fffffff;
            {
                const int32_t a0 = __shfl_sync(FULL, mlo, sx & 31);
                const int32_t b0 = __shfl_sync(FULL, mhi, sx & 31);
                if (sx >= 0 && a0 <= b0) {
                    ulo = a0;
                    uhi = b0;
                }
                const int32_t a1 = __shfl_sync(FULL, mlo, soe & 31);
                const int32_t b1 = __shfl_sync(FULL, mhi, soe & 31);
                if (soe >= 0 && a1 <= b1) {
                    ulo = min(ulo, a1 - 1);
                    uhi = max(uhi, b1 + 1);
                }
                const int32_t a2 = __shfl_sync(FULL, ilo, se & 31);
                const int32_t b2 = __shfl_sync(FULL, ihi, se & 31);
                if (se >= 0 && a2 <= b2) {  // I[s-e] at k-1 and D[s-e] at k+1
                    ulo = min(ulo, a2 - 1);
                    uhi = max(uhi, b2 + 1);
                }
            }
            const int32_t a = max(ulo, lo);
            const int32_t b = min(uhi, hi);
            ms = nms;
            is = nis;
            const int32_t omlo = __shfl_sync(FULL, mlo, ms);
            const int32_t omhi = __shfl_sync(FULL, mhi, ms);
            const int32_t oilo = __shfl_sync(FULL, ilo, is);
            const int32_t oihi = __shfl_sync(FULL, ihi, is);
            RT *const Mw = slot(ms);
            RT *const Iw = slot(hm + is);
            RT *const Dw = slot(hm + hie + is);
            // what the reused slots held outside [a, b] becomes NEG (all of it
            // when this score is empty)
            const int32_t ca = a > b ? 0x7fffffff : a, cb = a > b ? -0x7fffffff : b;
            if ((omlo <= omhi && (omlo < ca || omhi > cb)) ||
                (oilo <= oihi && (oilo < ca || oihi > cb))) {
                for (int32_t k = omlo + tt; k <= min(omhi, ca - 1); k += TW)
                    Mw[k] = (RT)NEG;
                for (int32_t k = max(omlo, cb + 1) + tt; k <= omhi; k += TW)
                    Mw[k] = (RT)NEG;
                for (int32_t k = oilo + tt; k <= min(oihi, ca - 1); k += TW) {
                    Iw[k] = (RT)NEG;
                    Dw[k] = (RT)NEG;
                }
                for (int32_t k = max(oilo, cb + 1) + tt; k <= oihi; k += TW) {
                    Iw[k] = (RT)NEG;
                    Dw[k] = (RT)NEG;
                }
            }
            bool hit = false;
            if (a <= b) {
                cells += (int64_t)(b - a + 1);
                // a source that does not exist yet reads the row kept NEG (slot nslot)
                const RT *negrow = slot(w.nslot);
                const RT *Mx = sx >= 0 ? slot(sx) : negrow;
                const RT *Moe = soe >= 0 ? slot(soe) : negrow;
                const RT *Ie = se >= 0 ? slot(hm + se) : negrow;
                const RT *De = se >= 0 ? slot(hm + hie + se) : negrow;
                // rounds of UU diagonals per thread: full rounds (every diagonal
                // inside [a, b]) while they last, then single-diagonal rounds
                auto round = [&](int32_t k0, auto uc, auto fc) {
                    constexpr int UU = decltype(uc)::value;
                    constexpr bool FULLR = decltype(fc)::value;
                    int32_t ks[UU], iv[UU], dv[UU], mv[UU];
                    bool live[UU];
#pragma unroll
                    for (int u = 0; u < UU; ++u) {
                        ks[u] = k0 + TW * u;
                        live[u] = FULLR || ks[u] <= b;
                        const int32_t kc = FULLR ? ks[u] : (live[u] ? ks[u] : b);
                        const int32_t io = (int32_t)Moe[kc - 1], dop = (int32_t)Moe[kc + 1];
                        const int32_t ie = (int32_t)Ie[kc - 1], dex = (int32_t)De[kc + 1];
                        const int32_t mx = (int32_t)Mx[kc];
                        const int32_t i0 = max(io, ie), d0 = max(dop, dex);
                        // max(mx + 1, i0 + 1, d0) as two DPX add-max instructions
                        const int32_t m1 = __viaddmax_s32(mx, 1, __viaddmax_s32(i0, 1, d0));
                        iv[u] = i0 < 0 ? NEG : i0 + 1;
                        mv[u] = m1 < 0 ? NEG : m1;
                        dv[u] = d0;
                    }
                    ext_u<UU, SMEM_SEQ>(qs, qlen, rs, rlen, mv, ks, live);
#pragma unroll
                    for (int u = 0; u < UU; ++u) {
                        if (live[u]) {
                            Iw[ks[u]] = (RT)iv[u];
                            Dw[ks[u]] = (RT)dv[u];
                            Mw[ks[u]] = (RT)mv[u];
                        }
                    }
                };
                int32_t k0 = a + tt;
                for (; k0 + TW * (U - 1) <= b; k0 += TW * U)
                    round(k0, std::integral_constant<int, U>{}, std::true_type{});
                for (; k0 <= b; k0 += TW)
                    round(k0, std::integral_constant<int, 1>{}, std::false_type{});
                // the thread that owns the target diagonal reads back its own store
                if ((uint32_t)(target - a) <= (uint32_t)(b - a) && ((target - a) & (TW - 1)) == tt)
                    hit = (int32_t)Mw[target] >= qlen;
            }
            if (lane == ms) {
                mlo = a <= b ? a : 1;
                mhi = a <= b ? b : 0;
            }
            if (lane == is) {
                ilo = a <= b ? a : 1;
                ihi = a <= b ? b : 0;
            }
            // M[s, target] >= qlen ends the alignment (:221-224)
            if (team.any(hit)) {
                result = s;
                break;
            }
        }
        if (result == kRunning)
            result = -1;  // the loop ran out: cost above max_error (:226)
    }
    return result;
}

// ---- tier kernel -----------------------------------------------------------------
// Work items: the pairs of `list` (int32 pair indices; nullptr = 0..n-1) or of
// `ents` ({pair, dump record or -1}); n from the host, or from *n_dev when
// set.  Items are handed out by atomics on ctr.
struct TierIn {
    const int32_t *list;
    const int2 *ents;
    int64_t n;
    const int *n_dev;
    const int64_t *seg;     // when set: list + seg[0], n = seg[1] - seg[0]
    int *ctr;
    const uint8_t *dumps;   // records the entries refer to
    int64_t dump_stride;
    const int32_t *ubound;  // per pair: a cost no lower than the optimum (-1: max_error)
    int32_t band_w;         // > 0: the bound pass's band half-width
};

struct TierOut {
    int2 *next;      // queue of the next tier
    int *next_n;
    DumpOut dump;    // records of pairs suspended here (base nullptr: none)
    int2 *restart;   // the G tier's queue
    int *restart_n;
};

struct TierGeom {
    int32_t W, H;           // window: elements per slot row, offset of diagonal 0
    int64_t team_bytes;     // shared bytes of one team (ring + sequence copies)
    int64_t ring_bytes;     // of them, the ring (shared) -- 0 for the G tier
    int32_t seq_cap;        // 16-base words per sequence copy, the guard's two included
    int32_t *gring;         // G tier: per-block int32 regions of nslot * W
};

template <int TEAM, int NTEAMS, typename RT, bool GRING>
__global__ void __launch_bounds__(TEAM *NTEAMS * 32, 1)
wfa_tier_kernel(SeqView q, SeqView r, WfaParams p, TierIn in, TierOut tout, TierGeom geo,
                int32_t *__restrict__ out, int64_t *work, int *err_flag)
{
    extern __shared__ __align__(16) uint8_t tsm[];
    __shared__ int64_t bcast[NTEAMS];
    const Shape w = make_shape(p);
    const int team_id = (int)(threadIdx.x / (TEAM * 32));
    const int tt = (int)(threadIdx.x % (TEAM * 32));
    const Team<TEAM, NTEAMS> team{team_id};
    uint8_t *const mine = tsm + team_id * geo.team_bytes;
    RT *ring;
    if (GRING)
        ring = reinterpret_cast<RT *>(geo.gring +
                                      (int64_t)blockIdx.x * (w.nslot + 1) * (int64_t)geo.W);
    else
        ring = reinterpret_cast<RT *>(mine);
    uint32_t *const sq = reinterpret_cast<uint32_t *>(mine + geo.ring_bytes);
    uint32_t *const sr = sq + geo.seq_cap;
    int64_t n = in.n;
    const int32_t *list = in.list;
    if (in.seg) {
        list = in.list + in.seg[0];
        n = in.seg[1] - in.seg[0];
    }
    if (in.n_dev)
        n = *in.n_dev;
    int64_t cells = 0;
    volatile int64_t *bc = &bcast[team_id];
    // A team's first item is given by its place in the grid, one team of every block
    // before the second of any: the longest pairs, first in the list, go to as many SMs
    // as there are.  Later ones are asked for.
    int64_t it = (int64_t)team_id * gridDim.x + blockIdx.x;
    for (bool asked = false;; asked = true) {
        if (asked) {
            if (tt == 0)
                *bc = atomicAdd(in.ctr, 1) + (int64_t)gridDim.x * NTEAMS;
            team.sync();
            it = *bc;
            team.sync();  // every thread has read the slot before it is reused
        }
        if (it >= n)
            break;
        int64_t pi;
        const uint8_t *resume = nullptr;
        if (in.ents) {
            const int2 e = in.ents[it];
            pi = e.x;
            if (e.y >= 0 && in.dumps)
                resume = in.dumps + (int64_t)e.y * in.dump_stride;
        } else {
            pi = list ? (int64_t)list[it] : it;
        }
        const int64_t ql = q.lengths[pi], rl = r.lengths[pi];
        const bool smem_seq = 2 * ((ql + 31) >> 5) + 2 <= geo.seq_cap &&  // and the guard
                              2 * ((rl + 31) >> 5) + 2 <= geo.seq_cap;
        int64_t di = -2;
        int32_t res;
        int32_t ub = -1;
        if (in.ubound) {
            ub = in.ubound[pi];
            if (ub < 0)
                ub = p.max_error;
        }
        auto align = [&](auto smem) -> int32_t {
            constexpr bool SMEM = decltype(smem)::value;
            if constexpr (GRING)
                return tier_pair32<TEAM, NTEAMS, 4, SMEM>(q, r, p, w, pi, ring, geo.W, geo.H, sq,
                                                          sr, team, cells, ub);
            else
                return tier_pair16<TEAM, NTEAMS, SMEM>(q, r, p, w, pi, ring, geo.W, geo.H, sq, sr,
                                                       team, bc, resume, tout.dump, &di, cells,
                                                       in.band_w, ub);
        };
        res = smem_seq ? align(std::true_type{}) : align(std::false_type{});
        if (tt == 0) {
            if (res >= -1) {
                out[pi] = res;
            } else if (res == kPromote && tout.next) {
                const int slot = atomicAdd(tout.next_n, 1);
                tout.next[slot] = make_int2((int)pi, (int)di);
            } else if (tout.restart) {
                // kRestart, or a window overflow with no tier above: the G tier
                const int slot = atomicAdd(tout.restart_n, 1);
                tout.restart[slot] = make_int2((int)pi, -1);
            } else if (in.band_w > 0) {
                out[pi] = -1;  // the bound pass could not finish this pair: no bound
            } else {
                out[pi] = -3;  // no tier left (the G window holds every diagonal)
                atomicOr(err_flag, 1);
            }
        }
    }
    if (tt == 0 && work && cells)
        atomicAdd((unsigned long long *)work, (unsigned long long)cells);
}

// ---- short pairs -------------------------------------------------------------------
// Batches whose longest sequence has at most kWfaShortLen bases start here: eight lanes
// per pair, four pairs per warp.  A read's wavefront is a dozen diagonals wide for a dozen
// steps, so a whole warp on it idles and repeats the per-step bookkeeping for one pair;
// here four pairs share it.  The slots rotate for the whole warp: a pair enters with its
// score 0 in the slot that is current, whatever step the others are at.  Nothing is pruned
// and the limits of the matrix only cut, so the diagonals of a pair's step sp are
// [max(-reach, -rlen), min(reach, qlen)] with a reach that depends on the penalties and sp
// alone: a table.  New pairs are taken when two of the four are done, so that their setup
// is shared.  A pair whose interval outgrows the window, or its steps the table, is queued
// for T1, which starts it over.  Blocks of four warps, five per SM.
// Bound: ALU issue (81% busy).  500,000 reads of 150 bp at up to 6% divergence: the call
// 2.91 -> 1.46 ms, the kernel 1.20 (T1 took 2.62); 1,800 warp instructions a pair against
// 3,600.  With the four pairs in step from their first to the last of them to end, 1.35.
struct ShortGeom {
    int32_t W, H, seq_cap;
    int32_t pair_bytes;
};
constexpr int kShortSteps = 512;

// reach[sp] = {of M; what the reused slots held}: the furthest diagonals of the pairs'
// step sp (-1: none) and of the steps whose slots it takes over.  By one thread.
__device__ void short_reach(const Shape &w, uchar2 *reach)
{
    int8_t rm[32], ri[32];  // per M slot: M, and I and D
    for (int j = 0; j < w.hm; ++j)
        rm[j] = ri[j] = -1;
    rm[0] = 0;
    int ms = 0;
    for (int sp = 1; sp < kShortSteps; ++sp) {
        ms = ms + 1 == w.hm ? 0 : ms + 1;
        auto back = [&](int d) { return ms >= d ? ms - d : ms - d + w.hm; };
        int vid = max(rm[back(w.oes)], ri[back(w.es)]);
        vid += vid >= 0;
        const int va = max(vid, (int)rm[back(w.xs)]);
        const int old = max((int)rm[ms], (int)ri[back(w.hie)]);
        reach[sp] = make_uchar2((unsigned char)(va + 1), (unsigned char)(old + 1));
        rm[ms] = (int8_t)min(va, 126);  // past every window
        ri[ms] = (int8_t)min(vid, 126);
    }
}

__global__ void __launch_bounds__(128, 5)
wfa_short_kernel(SeqView q, SeqView r, WfaParams p, TierIn in, int2 *next, int *next_n,
                 ShortGeom geo, int32_t *__restrict__ out, int64_t *work)
{
    extern __shared__ __align__(16) uint8_t tsm[];
    __shared__ uchar2 reach[kShortSteps];
    const unsigned FULL = 0xffffffffu;
    const Shape w = make_shape(p);
    const int lane = threadIdx.x & 31, sub = lane >> 3, l8 = lane & 7, warp = threadIdx.x >> 5;
    const int32_t W = geo.W, H = geo.H;
    const int hm = w.hm, hie = w.hie, xs = w.xs, oes = w.oes, es = w.es;
    uint8_t *const mine = tsm + (warp * 4 + sub) * geo.pair_bytes;
    int16_t *const ring = reinterpret_cast<int16_t *>(mine);
    uint32_t *const sq = reinterpret_cast<uint32_t *>(mine + w.nslot * W * 2);
    uint32_t *const sr = sq + geo.seq_cap;
    if (threadIdx.x == 0)
        short_reach(w, reach);
    __syncthreads();
    int64_t n = in.n;
    const int32_t *list = in.list;
    if (in.seg) {
        list = in.list + in.seg[0];
        n = in.seg[1] - in.seg[0];
    }
    const int32_t sp_end = p.max_error / w.g;
    const int32_t mrows = hm * W, irows = hie * W;
    int64_t cells = 0;
    // the warp's slots
    int ms = 0, is = 0;
    int32_t om = 0, oi = 0;
    // this lane's pair
    bool active = false;
    int32_t pi = 0, qlen = 0, rlen = 0, target = 0, sp = 0;
    uint32_t qguard2 = 0, rguard2 = 0;
    const SeqWin qs{sq, nullptr, 0}, rs{sr, nullptr, 0};
    // pairs come four (then as many as are done) at a time: the first by the warp's place
    int64_t given = ((int64_t)warp * gridDim.x + blockIdx.x) * 4;
    bool more = true, asked = false;
    for (;;) {
        const unsigned act = __ballot_sync(FULL, active) & 0x01010101u;
        const int idle = 4 - __popc(act);
        if (more && idle >= 2) {
            if (asked) {
                int64_t b0 = 0;
                if (lane == 0)
                    b0 = atomicAdd(in.ctr, idle) + (int64_t)gridDim.x * 16;
                given = __shfl_sync(FULL, b0, 0);
            }
            asked = true;
            const int64_t it =
                given + __popc(~act & 0x01010101u & ((1u << (8 * sub)) - 1u));
            more = given + idle < n;
            const bool fresh = !active && it < n;
            if (fresh) {
                pi = list ? list[it] : (int32_t)it;
                qlen = (int32_t)q.lengths[pi];
                rlen = (int32_t)r.lengths[pi];
                const int32_t qnw = (qlen + 31) >> 5, rnw = (rlen + 31) >> 5;
                stage_seq<true>(q, q.offsets[pi] - q.word_base, qnw, sq, l8, 8, 0u);
                stage_seq<true>(r, r.offsets[pi] - r.word_base, rnw, sr, l8, 8, 0xFFFFFFFFu);
                uint4 *v = reinterpret_cast<uint4 *>(ring);
                const uint4 n4 = make_uint4(0x80008000u, 0x80008000u, 0x80008000u, 0x80008000u);
                for (int32_t i = l8; i < w.nslot * W / 8; i += 8)
                    v[i] = n4;
                target = qlen - rlen;
                qguard2 = (uint32_t)qnw * 64u;
                rguard2 = (uint32_t)rnw * 64u;
            }
            __syncwarp();
            if (fresh) {
                // score 0: M[0,0] = 0 extended along diagonal 0 (:130-140)
                const int32_t row0 = ext_more<true>(qs, qlen, rs, rlen, 0, 0);
                sp = 0;
                active = !(target == 0 && row0 >= qlen) && sp_end > 0;
                if (l8 == 0) {
                    ring[om + H] = (int16_t)row0;
                    cells += 1;
                    if (!active)
                        out[pi] = target == 0 && row0 >= qlen ? 0 : -1;
                }
            }
            __syncwarp();
            continue;
        }
        if (!act)
            break;
        // one step of every pair
        ++sp;
        ms = ms + 1 == hm ? 0 : ms + 1;
        is = is + 1 == hie ? 0 : is + 1;
        om = om + W == mrows ? 0 : om + W;
        oi = oi + W == irows ? 0 : oi + W;
        const int32_t ox = om >= xs * W ? om - xs * W : om - xs * W + mrows;
        const int32_t ooe = om >= oes * W ? om - oes * W : om - oes * W + mrows;
        const int32_t oe = oi >= es * W ? oi - es * W : oi - es * W + irows;
        int16_t *const Mw = ring + om, *const Iw = ring + mrows + oi, *const Dw = Iw + irows;
        int32_t va = -1;
        if (active) {
            const uchar2 re = reach[min(sp, kShortSteps - 1)];
            va = (int32_t)re.x - 1;
            // what the reused slots held further out, inside the window, becomes NEG
            for (int k = va + 1 + l8; k <= min((int)re.y - 1, H); k += 8) {
                Mw[H + k] = Iw[H + k] = Dw[H + k] = (int16_t)-32768;
                Mw[H - k] = Iw[H - k] = Dw[H - k] = (int16_t)-32768;
            }
        }
        const int32_t a = max(-va, -rlen), b = min(va, qlen);
        if (active && (a - 4 < -H || b + 5 > W - 1 - H || sp >= kShortSteps - 1)) {
            active = false;
            if (l8 == 0)
                next[atomicAdd(next_n, 1)] = make_int2(pi, -1);
        }
        const int32_t pa = H + a, pb = active && va >= 0 ? H + b : -1;
        if (l8 == 0)
            cells += max(pb - pa + 1, 0);
        const int16_t *const Mx = ring + ox, *const Moe = ring + ooe, *const Ie = ring + mrows + oe;
        const int16_t *const De = Ie + irows;
        // one round of two diagonals a lane covers 16 positions from an even one; wider
        // intervals take rounds of four
        if (__any_sync(FULL, pb - (pa & ~1) >= 16)) {
            for (int32_t at = (pa & ~3) + 4 * l8; __any_sync(FULL, at <= pb); at += 32)
                if (at <= pb)
                    wf_group<4, true>(Mx, Moe, Ie, De, Mw, Iw, Dw, at, at - H, pa, pb, qs, qlen,
                                      rs, rlen, qguard2, rguard2);
        } else {
            const int32_t at = (pa & ~1) + 2 * l8;
            if (at <= pb)
                wf_group<2, true>(Mx, Moe, Ie, De, Mw, Iw, Dw, at, at - H, pa, pb, qs, qlen, rs,
                                  rlen, qguard2, rguard2);
        }
        __syncwarp();
        // M[s, target] >= qlen ends the alignment (:221-224)
        const bool hit = pb >= 0 && a <= target && target <= b && (int32_t)Mw[H + target] >= qlen;
        if (active && (hit || sp >= sp_end)) {
            active = false;
            if (l8 == 0)
                out[pi] = hit ? sp * w.g : -1;
        }
    }
    if (l8 == 0 && work && cells)
        atomicAdd((unsigned long long *)work, (unsigned long long)cells);
}

}  // namespace

// ---- host side --------------------------------------------------------------------
// Shared memory of one block (the device maximum per block, less a margin for
// the kernel's static shared variables).
constexpr int64_t kTierBlockSmem = 227 * 1024 - 256;
constexpr int64_t kTierMinWindow = 64;  // diagonals

struct TierSpec {
    int team_warps, nteams;
    int32_t seq_bases;  // longest sequence copied to shared memory
};
// S, M, L tiers
static const TierSpec kTiers[kWfaShared] = {{1, 16, kWfaOneWarpCopy}, {2, 8, 12288}, {4, 4, 16384}, {8, 2, 32768}, {16, 1, 32768}};

WfaTierPlan wfa_tier_plan(const WfaParams &p, int64_t qmax, int64_t rmax)
{
    auto gcd_h = [](int a, int b) {
        while (b) {
            const int t = a % b;
            a = b;
            b = t;
        }
        return a;
    };
    const int g = gcd_h(p.x, gcd_h(p.o, p.e));
    const int hm = std::max(p.x / g, (p.o + p.e) / g) + 1, hie = p.e / g + 1;
    const int nslot = hm + 2 * hie;
    WfaTierPlan plan{};
    plan.nslot = nslot;
    for (int t = 0; t < kWfaShared; ++t) {
        const TierSpec &s = kTiers[t];
        const int64_t team_bytes = kTierBlockSmem / s.nteams;
        int64_t seq_entries = 2 * ((s.seq_bases + 31) / 32) + 2;  // and the guard
        int64_t W = (team_bytes - 2 * seq_entries * 4) / (nslot * 2);
        W = W / 8 * 8;  // 16-byte rows: the NEG fill uses 16-byte stores
        // Many slots (up to 96) leave the one-warp tier less than 64 diagonals: it keeps 64
        // and copies shorter sequences (x1 o0 e31, 400,000 pairs of 100 bp: 126 ms without
        // that tier, 96 so).
        if (W < kTierMinWindow && team_bytes > kTierMinWindow * nslot * 2) {
            const int64_t words = (team_bytes - kTierMinWindow * nslot * 2) / 8 & ~int64_t(1);
            if (words >= 4) {
                W = kTierMinWindow;
                seq_entries = std::min(seq_entries, words);
            }
        }
        plan.W[t] = (int32_t)W;
        plan.H[t] = (int32_t)(W / 2 - 1);
        plan.seq_cap[t] = (int32_t)seq_entries;
        plan.team_bytes[t] = team_bytes & ~int64_t(15);
        plan.ring_bytes[t] = (int64_t)nslot * W * 2;
        plan.usable[t] = W >= kTierMinWindow;
        plan.dump_stride[t] = (kDumpHeader + (int64_t)nslot * W * 2 + 255) & ~int64_t(255);
    }
    // G: int32 rings covering [-max(qlen, rlen) - 3, max(qlen, rlen) + 3]
    const int64_t lmax = std::max(qmax, rmax);
    constexpr int G = kWfaShared;
    plan.W[G] = (int32_t)(((2 * lmax + 8) + 7) & ~int64_t(7));
    plan.H[G] = (int32_t)(lmax + 3);
    plan.seq_cap[G] = (int32_t)(2 * ((kTiers[G - 1].seq_bases + 31) / 32) + 2);
    plan.team_bytes[G] = 2 * (int64_t)plan.seq_cap[G] * 4;
    plan.ring_bytes[G] = 0;
    plan.usable[G] = true;
    plan.gring_block_bytes = (int64_t)(nslot + 1) * plan.W[G] * 4;
    return plan;
}

// Shared memory of a pair of the short kernel: five blocks of sixteen pairs per SM, and
// the pairs' rows half a set of banks apart, so that four pairs' 8-byte loads of the same
// row fall on both halves.
constexpr int32_t kShortPairBytes = 2752;
static_assert(kShortPairBytes % 128 == 64 &&
                  5 * (16 * kShortPairBytes + kSeqSlack + 2 * kShortSteps + 1024) <= 228 * 1024,
              "five blocks per SM");

static ShortGeom short_geom(int nslot)
{
    ShortGeom g;
    g.seq_cap = 2 * ((kWfaShortLen + 31) / 32) + 2;
    g.W = (kShortPairBytes - 8 * g.seq_cap) / (nslot * 2) / 8 * 8;
    g.W = std::min(g.W, 248);  // the reach table's bytes
    g.H = g.W / 2 - 1;
    g.pair_bytes = kShortPairBytes;
    return g;
}

bool wfa_short_usable(const WfaTierPlan &pl) { return short_geom(pl.nslot).W >= 64; }

cudaError_t launch_wfa_short(const WfaTierPlan &pl, int sm_count, SeqView q, SeqView r, WfaParams p,
                             const WfaTierIo &io, int32_t *out, int64_t *work, cudaStream_t st)
{
    static std::atomic<uint64_t> smem_set{0};
    const cudaError_t attr =
        allow_smem(wfa_short_kernel, 16 * kShortPairBytes + kSeqSlack, smem_set);
    if (attr != cudaSuccess)
        return attr;
    TierIn in{};
    in.list = io.list;
    in.n = io.n;
    in.seg = io.seg;
    in.ctr = io.ctr;
    const int grid = (int)std::min<int64_t>(5 * (int64_t)sm_count, (io.n + 15) / 16);
    wfa_short_kernel<<<grid, 128, 16 * kShortPairBytes + kSeqSlack, st>>>(q, r, p, in, io.next, io.next_n,
                                                               short_geom(pl.nslot), out, work);
    return cudaGetLastError();
}

template <int TEAM, int NTEAMS, typename RT, bool GRING>
static cudaError_t tier_launch(const WfaTierPlan &pl, int t, int grid, SeqView q, SeqView r,
                               WfaParams p, const TierIn &in, const TierOut &o, int32_t *gring,
                               int32_t *out, int64_t *work, int *err_flag, cudaStream_t st)
{
    const size_t smem = (size_t)pl.team_bytes[t] * NTEAMS + kSeqSlack;
    static std::atomic<uint64_t> smem_set{0};
    const cudaError_t attr = allow_smem(wfa_tier_kernel<TEAM, NTEAMS, RT, GRING>,
                                        (int)kTierBlockSmem + kSeqSlack, smem_set);
    if (attr != cudaSuccess)
        return attr;
    TierGeom geo{pl.W[t], pl.H[t], pl.team_bytes[t], pl.ring_bytes[t], pl.seq_cap[t], gring};
    wfa_tier_kernel<TEAM, NTEAMS, RT, GRING><<<grid, TEAM * NTEAMS * 32, smem, st>>>(
        q, r, p, in, o, geo, out, work, err_flag);
    return cudaGetLastError();
}

cudaError_t launch_wfa_tier(const WfaTierPlan &pl, int tier, int grid, SeqView q, SeqView r,
                            WfaParams p, const WfaTierIo &io, int32_t *out, int64_t *work,
                            int *err_flag, cudaStream_t st)
{
    TierIn in{io.list,    io.ents,           io.n,      io.n_dev, io.seg,
              io.ctr,     io.dumps_in,       io.dump_in_stride,   io.ubound, io.band_w};
    TierOut o{io.next, io.next_n, DumpOut{io.dumps_out, io.dump_out_stride, io.dump_out_cap,
                                          io.dump_out_ctr},
              io.restart, io.restart_n};
    switch (tier) {
    case 0:
        return tier_launch<1, 16, int16_t, false>(pl, 0, grid, q, r, p, in, o, nullptr, out,
                                                  work, err_flag, st);
    case 1:
        return tier_launch<2, 8, int16_t, false>(pl, 1, grid, q, r, p, in, o, nullptr, out,
                                                 work, err_flag, st);
    case 2:
        return tier_launch<4, 4, int16_t, false>(pl, 2, grid, q, r, p, in, o, nullptr, out,
                                                 work, err_flag, st);
    case 3:
        return tier_launch<8, 2, int16_t, false>(pl, 3, grid, q, r, p, in, o, nullptr, out,
                                                 work, err_flag, st);
    case 4:
        return tier_launch<16, 1, int16_t, false>(pl, 4, grid, q, r, p, in, o, nullptr, out,
                                                  work, err_flag, st);
    default:
        return tier_launch<16, 1, int32_t, true>(pl, kWfaShared, grid, q, r, p, in, o, io.gring,
                                                 out, work, err_flag, st);
    }
}

}  // namespace gb2
