// xw_packed.cuh -- one annealing iteration on packed rows, for orders up to
// 128: the device code shared by the one-warp replica loop and the latency
// mode of xw_anneal.cu.
//
// W and its Gram matrix sit in the replica's shared-memory slot as biased
// bytes, four rows of a column of W (or four entries of a row of G) to a
// 32-bit word: w + 1 and G + 128, with G's diagonal kept at 0.  Every move
// changes at most two rows of W, in at most the two columns C1 and C2, so a
// changed Gram row is
//   G'[R] = G[R] + a W[:,C1] + b W[:,C2],
// and because the bias makes every byte an unsigned digit in base 256, that
// sum is two multiply-adds on whole words: four entries a time, no carries
// between bytes (new entries stay within +-127).  The score of a row is the
// sum of |G| over its bytes (vabsdiff4 against 128, dp4a) and its conflicts
// the count of nonzero ones; both are kept per row (the packed residual), so
// an evaluation reads only the new values.
//
// A group of LPC lanes (8 of a warp, 4 of a half-warp) works on one
// candidate move from its draws to its deltas: the lanes share the hot-row
// tournament, each computes the proposal (the same instructions for all
// four groups), and each evaluates its own 4*WPL rows.  The group's sums
// come together in log2(LPC) shuffles and the best candidate in one
// warp-wide minimum of a key that orders by (deltas, candidate).  Four
// candidates therefore cost one pass: 4x fewer instructions than a loop
// over candidates with one row per lane.
//
// What bounds it: instruction issue of dependent integer chains.  Measured
// on B200 against a loop over candidates with one row per lane and a 32-bit
// Gram matrix: 593 warp instructions an iteration against 843 (W(26,25)
// ladder, 10^4 iterations of 4096 replicas: 30.5 ms against 44.7); W(100,50),
// 592 replicas of 1000 iterations: 5.6 ms against 13.5 (bytes let six warps
// share an SM instead of three, and the group's lanes try the attempts of a
// support switch eight at a time).
#pragma once

#include <cuda_runtime.h>

#include "xw_device.cuh"
#include "xw_kernels.h"

namespace xw {

extern __shared__ __align__(16) uint8_t xw_smem[];

namespace {

constexpr unsigned FULL = 0xffffffffu;

// Lane groups.  A replica is owned by a group of GW lanes: the whole warp
// (GW = 32), or one half of it (GW = 16, orders up to 16: two replicas per
// warp, each half with its own shared-memory slot and its own work items).
// Warp collectives name only the group's lanes; the two halves' replicas
// are independent and the hardware runs them side by side wherever their
// control flow agrees.
template <int GW>
__device__ __forceinline__ unsigned group_mask() {
    if constexpr (GW == 32) return FULL;
    else return 0xffffu << (threadIdx.x & 16);
}

// Metropolis thresholds kept per replica for objective increases 1..kThrTable.
constexpr uint32_t kThrTable = 64;

__device__ __forceinline__ int iabs(int v) { return v < 0 ? -v : v; }

__device__ __forceinline__ uint32_t lds8(uint32_t a) { return xw_smem[a]; }
__device__ __forceinline__ uint32_t lds32(uint32_t a) { return *reinterpret_cast<const uint32_t*>(xw_smem + a); }
__device__ __forceinline__ uint4 lds128(uint32_t a) { return *reinterpret_cast<const uint4*>(xw_smem + a); }
__device__ __forceinline__ uint64_t lds64(uint32_t a) { return *reinterpret_cast<const uint64_t*>(xw_smem + a); }

// Bytes from one column of W (row of G) to the next: a multiple of the
// 4*WPL bytes a lane reads at once, and an odd multiple, so that the
// mirrored column of a commit, one byte in each row, spreads over the banks.
__host__ __device__ constexpr uint32_t packed_stride(int n, int wpl) {
    const uint32_t q = 4u * (uint32_t)wpl;
    return ((((uint32_t)n + q - 1u) / q) | 1u) * q;
}

// Replica constants read by broadcast from the slot.
struct Con {
    uint64_t thr_target, thr_dbl, thr_sign, thr_swsign;
    uint64_t thr_greedy;
    double T;
};

// The slot: fixed regions first, so that their offsets are constants.
template <int WPL>
struct Slot {
    static constexpr uint32_t draws = 0;                      // 32 Philox blocks
    static constexpr uint32_t thr = 512;                      // Metropolis thresholds
    static constexpr uint32_t con = thr + 8u * kThrTable;
    static constexpr uint32_t res = con + 64u;                // packed residuals, 4 bytes a row
    static constexpr uint32_t mask = res + 128u * WPL;        // support masks, 4*WPL bytes a row
    static constexpr uint32_t w = mask + 128u * WPL * WPL;
};

static_assert(sizeof(Con) <= 64, "replica constants fit their region");

__host__ __device__ constexpr uint32_t packed_slot_bytes(int n, int m, int wpl) {
    const uint32_t fixed = 512u + 8u * kThrTable + 64u + 128u * (uint32_t)wpl + 128u * (uint32_t)(wpl * wpl);
    const uint32_t mat = xw_pad16((uint32_t)n * packed_stride(n, wpl));
    // the last lanes of a row may read up to one lane's width past it; the
    // minority lists' pad covers the read of an empty list
    return fixed + 2u * mat + xw_pad16((uint32_t)(n * m) + 1u);
}

// Loop-invariant context of a replica's lane group.
struct Env {
    uint32_t slot;       // the replica's slot in xw_smem
    uint32_t draws;      // this group's draw buffer
    uint32_t g, mino;    // byte offsets of G and the minority lists
    uint32_t st;         // row stride
    int n, w, m, sparse;
    uint32_t k0, k1, stream;
    int cs, ts, bpc, move_set, obj_kind;
    uint32_t my_slot, my_slot2;   // Philox counter slots of this lane's cached blocks
    uint32_t loff;       // byte offset of the lane's rows
    int l, grp;          // lane within its candidate, candidate within a pass
    bool lact;           // the lane holds rows below n
};

// ---- proposals --------------------------------------------------------

__device__ __forceinline__ int first_from(uint32_t m, int start) {
    const uint32_t hi = m & (0xffffffffu << start);
    return __ffs((int)(hi ? hi : m)) - 1;
}

__device__ __forceinline__ int first_from(uint64_t m, int start) {
    const uint64_t hi = m & (~0ull << start);
    return __ffsll((long long)(hi ? hi : m)) - 1;
}

// First set bit at or after `start`, cyclically, of row `row`'s support
// mask (COMPL: of its complement below n).
template <int WPL, bool COMPL = false>
__device__ __forceinline__ int mask_first(uint32_t slot, int row, int start, int n) {
    const uint32_t a = slot + Slot<WPL>::mask + (uint32_t)row * (4u * WPL);
    if constexpr (WPL == 1) {
        uint32_t m = lds32(a);
        if (COMPL) m = ~m & (n >= 32 ? 0xffffffffu : (1u << n) - 1u);
        return first_from(m, start);
    } else if constexpr (WPL == 2) {
        uint64_t m = lds64(a);
        if (COMPL) m = ~m & (n >= 64 ? ~0ull : (1ull << n) - 1ull);
        return first_from(m, start);
    } else {
        uint64_t lo = lds64(a), hi = lds64(a + 8);
        if (COMPL) {
            lo = ~lo;
            hi = ~hi & (n >= 128 ? ~0ull : (1ull << (n - 64)) - 1ull);
        }
        // rotate so that the search starts in the first word
        if (start >= 64) {
            const uint64_t h = hi & (~0ull << (start - 64));
            if (h) return 64 + __ffsll((long long)h) - 1;
            if (lo) return __ffsll((long long)lo) - 1;
            return 64 + __ffsll((long long)hi) - 1;
        }
        const uint64_t h = lo & (~0ull << start);
        if (h) return __ffsll((long long)h) - 1;
        if (hi) return 64 + __ffsll((long long)hi) - 1;
        return __ffsll((long long)lo) - 1;
    }
}

// A draw word outside the cached blocks (tournaments past 8 samples).
__device__ __noinline__ uint32_t slow_word(uint32_t slot, uint64_t it, uint32_t stream, uint32_t k0, uint32_t k1,
                                           int j) {
    return pick(draw_block(slot, it, stream, k0, k1), j);
}

// Column of a sign flip in `row` from draw word `wd` (slot, word j of block
// b), propose_sign_flip (xweigh_cuda.cu:302-325): a minority pick for a
// sparse row, else the first nonzero at or after a random column.
template <int WPL>
__device__ __forceinline__ int flip_col_exact(uint32_t slot, uint32_t mino, int n, int m, int sparse, uint32_t wd,
                                              uint32_t dslot, uint64_t it, uint32_t stream, uint32_t k0, uint32_t k1,
                                              int j, int row) {
    if (sparse && m > 0) return (int)lds8(mino + (uint32_t)(row * m) + draw_index(wd, (uint32_t)m, dslot, it, stream, k0, k1, j));
    return mask_first<WPL>(slot, row, (int)draw_index(wd, (uint32_t)n, dslot, it, stream, k0, k1, j), n);
}

// The whole proposal of candidate `c` with exact index draws and every
// further attempt, propose_move (xweigh_cuda.cu:327-447): called by the
// groups whose first attempt is not legal (a second flip that repeats the
// first, a switch whose 2x2 is not legal) or whose draws met Lemire's
// rejection zone.  Attempts are independent given their counters, so the
// group's lanes try LPC of them at once and the first legal one is taken;
// in order this is one attempt after the other, each with its own Philox
// block.  `need`: the calling lane's group wants a proposal (the other
// lanes take part in the collectives only).  Returns
// {R1 | R2<<8 | C1<<16 | C2<<24, kind | p1<<8 | p2<<16 | s1<<24 | s2<<25}.
template <int WPL, int GW>
__device__ __noinline__ uint2 propose_exact(bool need, uint32_t slot, uint32_t cw, uint32_t mino, uint32_t st, int n,
                                            int w, int m, int sparse, int hot, int c, uint64_t it, uint32_t stream,
                                            uint32_t k0, uint32_t k1) {
    constexpr int LPC = GW / 4;
    const unsigned gm = group_mask<GW>();
    const int wl = threadIdx.x & 31, l = wl & (LPC - 1), base = wl - l;
    const Con* con = reinterpret_cast<const Con*>(xw_smem + slot + Slot<WPL>::con);
    const uint4 b0 = lds128(cw), b1 = lds128(cw + 16), b2 = lds128(cw + 32), b3 = lds128(cw + 48);
    auto ix = [&](uint32_t wd, uint32_t count, int b, int j) -> int {
        return (int)draw_index(wd, count, cand_slot(c, b), it, stream, k0, k1, j);
    };
    auto fcol = [&](uint32_t wd, int b, int j, int row) -> int {
        return flip_col_exact<WPL>(slot, mino, n, m, sparse, wd, cand_slot(c, b), it, stream, k0, k1, j, row);
    };
    int row = 0, r2 = 0, c1 = 0, c2 = 0, p1 = 0, p2 = 0, kind = -1;
    bool s1 = false, s2 = false, dbl = false, flip = false;
    if (need) {
        row = (uint64_t)b0.x < con->thr_target ? hot : ix(b0.y, (uint32_t)n, 0, 1);
        dbl = (uint64_t)b0.z < con->thr_dbl;
        flip = w == n || (uint64_t)b0.w < con->thr_sign;
    }
    // double flip (xweigh_cuda.cu:389-421): attempt 0 from block 3, attempt
    // a > 0 from block 19 + a, 16 in all
    bool pend = need && dbl;
    if (__any_sync(gm, pend)) {
        const int first = pend ? fcol(b2.w, 2, 3, row) : 0;
#pragma unroll 1
        for (int a0 = 0; a0 < 16; a0 += LPC) {
            const int a = a0 + l;
            int rr = 0, cc = 0;
            bool ok = false;
            if (pend && a < 16) {
                const int b = a == 0 ? 3 : 19 + a;
                const uint4 d = a == 0 ? b3 : draw_block(cand_slot(c, b), it, stream, k0, k1);
                rr = d.x < 0x80000000u ? row : ix(d.y, (uint32_t)n, b, 1);
                cc = fcol(d.z, b, 2, rr);
                ok = !(rr == row && cc == first);
            }
            const unsigned hit = (__ballot_sync(gm, ok) >> base) & ((1u << LPC) - 1u);
            const int src = hit ? base + __ffs((int)hit) - 1 : wl;
            rr = __shfl_sync(gm, rr, src);
            cc = __shfl_sync(gm, cc, src);
            if (pend && hit) {
                kind = 2;
                r2 = rr;
                c1 = first;
                c2 = cc;
                pend = false;
            }
            if (!__any_sync(gm, pend)) break;
        }
    }
    if (need && kind < 0 && flip) {
        kind = 0;
        r2 = row;
        c1 = c2 = fcol(b1.x, 1, 0, row);
    }
    // support switch (xweigh_cuda.cu:327-387): attempt 0 in blocks 1 and 2,
    // attempt a > 0 in blocks 36 + 2(a-1) and the next, 24 in all
    pend = need && kind < 0 && m > 0 && n > 1;
    if (__any_sync(gm, pend)) {
#pragma unroll 1
        for (int a0 = 0; a0 < 24; a0 += LPC) {
            const int a = a0 + l;
            int rr = 0, x1 = 0, x2 = 0, q = 0, qq = 0;
            uint32_t sw1 = 0;
            bool ok = false;
            if (pend) {
                const int b = a == 0 ? 1 : 36 + 2 * (a - 1), o = a == 0 ? 1 : 0;
                const uint4 d = a == 0 ? make_uint4(b1.y, b1.z, b1.w, b2.x)
                                       : draw_block(cand_slot(c, b), it, stream, k0, k1);
                rr = ix(d.x, (uint32_t)(n - 1), b, o);
                if (rr >= row) ++rr;
                q = ix(d.y, (uint32_t)m, b, o + 1);
                qq = ix(d.z, (uint32_t)m, b, o + 2);
                sw1 = d.w;
                const int q1 = (int)lds8(mino + (uint32_t)(row * m + q)), q2 = (int)lds8(mino + (uint32_t)(rr * m + qq));
                x1 = sparse ? q1 : q2;
                x2 = sparse ? q2 : q1;
                // entries (row, x2) and (rr, x1) are zeros and (row, x1),
                // (rr, x2) nonzeros: one pair by the choice of q1, q2
                const uint32_t e1 = lds8(slot + Slot<WPL>::w + (uint32_t)q2 * st + (uint32_t)row);
                const uint32_t e2 = lds8(slot + Slot<WPL>::w + (uint32_t)q1 * st + (uint32_t)rr);
                ok = sparse ? e1 == 1u && e2 == 1u : e1 != 1u && e2 != 1u;
            }
            const unsigned hit = (__ballot_sync(gm, ok) >> base) & ((1u << LPC) - 1u);
            const int src = hit ? base + __ffs((int)hit) - 1 : wl;
            rr = __shfl_sync(gm, rr, src);
            x1 = __shfl_sync(gm, x1 | (x2 << 8) | (q << 16) | (qq << 24), src);
            sw1 = __shfl_sync(gm, sw1, src);
            if (pend && hit) {
                const int win = a0 + (src - base);
                kind = 1;
                r2 = rr;
                c1 = x1 & 255;
                c2 = (x1 >> 8) & 255;
                p1 = (x1 >> 16) & 255;
                p2 = (int)((uint32_t)x1 >> 24);
                s1 = (uint64_t)sw1 < con->thr_swsign;
                const uint32_t sw2 =
                    win == 0 ? b2.y : pick(draw_block(cand_slot(c, 36 + 2 * (win - 1) + 1), it, stream, k0, k1), 0);
                s2 = (uint64_t)sw2 < con->thr_swsign;
                pend = false;
            }
            if (!__any_sync(gm, pend)) break;
        }
    }
    if (need && kind < 0) {
        kind = 0;
        r2 = row;
        c1 = c2 = fcol(b2.z, 2, 2, row);
    }
    return make_uint2((uint32_t)row | ((uint32_t)r2 << 8) | ((uint32_t)c1 << 16) | ((uint32_t)c2 << 24),
                      (uint32_t)(kind & 3) | ((uint32_t)p1 << 8) | ((uint32_t)p2 << 16) | (s1 ? 1u << 24 : 0u) |
                          (s2 ? 1u << 25 : 0u));
}

// A move in three words:
//   rc  R1 | R2<<8 | C1<<16 | C2<<24 (R2 = R1: one row)
//   cf  the coefficients a1, b1 (row R1, columns C1, C2), a2, b2 (row R2)
//   ax  change of G[R1][R2] | p1<<8 | p2<<16 | support change<<24 (bit 0 R1,
//       bit 1 R2), p1, p2 the changed entries of the minority lists
struct Move {
    uint32_t rc, cf, ax;
};

// The move an iteration puts to the Metropolis test: the first best of its
// candidates, its deltas and the iteration's acceptance draw.  `mv` is the
// move of the lane's own candidate until it is taken from lane `src`.
struct Pick {
    Move mv;
    int src;
    int ds, dc, prim;
    uint32_t u;
};

template <int WPL>
__device__ __forceinline__ void load_words(uint32_t a, uint32_t (&v)[WPL]) {
    if constexpr (WPL == 1) {
        v[0] = lds32(a);
    } else if constexpr (WPL == 2) {
        const uint2 t = *reinterpret_cast<const uint2*>(xw_smem + a);
        v[0] = t.x; v[1] = t.y;
    } else {
        const uint4 t = lds128(a);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
}

// packed residual of a row: sum |G| | conflicts << 18
constexpr int kConfShift = 18;

// Iteration `it` against the replica's current state: draws, hot-row
// tournaments, proposals, evaluation.  Reads the state and writes only the
// group's draw buffer.  cand_l counts the candidates this lane's group
// evaluated, two_l those that change two rows.
template <int WPL, bool GEN, int GW, bool ONEZ>
__device__ __forceinline__ Pick choose(const Env& E, uint64_t it, int lane, uint32_t& cand_l, uint32_t& two_l) {
    constexpr int LPC = GW / 4;
    const unsigned gm = group_mask<GW>();
    const int n = E.n, m = ONEZ ? 1 : E.m, sparse = ONEZ ? 0 : E.sparse;
    const uint32_t st = E.st, slot = E.slot, wbase = E.slot + Slot<WPL>::w;
    const Con* con = reinterpret_cast<const Con*>(xw_smem + slot + Slot<WPL>::con);
    Pick P;
    P.src = 0;
    P.ds = P.dc = P.prim = 0;
    P.mv = Move{0, 0, 0};
    // A: draws (block 0 the move-level block, 1 + c*bpc + b block b of
    // candidate c; a half-warp computes two blocks per lane)
    uint4* dbuf = reinterpret_cast<uint4*>(xw_smem + E.draws);
    dbuf[lane] = draw_block(E.my_slot, it, E.stream, E.k0, E.k1);
    if constexpr (GW == 16) dbuf[lane + 16] = draw_block(E.my_slot2, it, E.stream, E.k0, E.k1);
    __syncwarp(gm);
    const uint64_t mblk = lds64(E.draws);
    P.u = (uint32_t)(mblk >> 32);
    const int count = (uint64_t)(uint32_t)mblk < con->thr_greedy ? E.cs : 1;
    uint32_t bestA = 0xffffffffu, bestB = 0xffffffffu;
    const uint32_t cw = E.draws + 16u + (uint32_t)(E.grp * E.bpc) * 16u;

#pragma unroll 1
    for (int c0 = 0;;) {
        const int c = c0 + E.grp;
        const bool act = c < count;
        // C: hot-row tournament (hot_row, xweigh_cuda.cu:291-300): the
        // first sample with the largest residual
        uint32_t key = 0;
        if (GW == 32 && E.ts <= 8) {
            if (E.l < E.ts) {
                const uint32_t r = draw_index(lds32(cw + 64u + 4u * (uint32_t)E.l), (uint32_t)n,
                                              cand_slot(c, 4 + (E.l >> 2)), it, E.stream, E.k0, E.k1, E.l & 3);
                key = (lds32(slot + Slot<WPL>::res + 4u * r) << 14) | ((uint32_t)(63 - E.l) << 8) | r;
            }
        } else {
#pragma unroll 1
            for (int s = E.l; s < E.ts; s += LPC) {
                const uint32_t ds = cand_slot(c, 4 + (s >> 2));
                const uint32_t wd = s < 8 ? lds32(cw + 64u + 4u * (uint32_t)s) : slow_word(ds, it, E.stream, E.k0, E.k1, s & 3);
                const uint32_t r = draw_index(wd, (uint32_t)n, ds, it, E.stream, E.k0, E.k1, s & 3);
                key = max(key, (lds32(slot + Slot<WPL>::res + 4u * r) << 14) | ((uint32_t)(63 - s) << 8) | r);
            }
        }
#pragma unroll
        for (int d = 1; d < LPC; d <<= 1) key = max(key, __shfl_xor_sync(gm, key, d));
        const int hot = (int)(key & 255u);

        // D: the first attempt of the proposal (propose_move,
        // xweigh_cuda.cu:423-447)
        const uint4 b0 = lds128(cw), b1 = lds128(cw + 16), b2 = lds128(cw + 32), b3 = lds128(cw + 48);
        bool edge = false;   // a draw met Lemire's rejection test: take the exact proposal
        auto ix = [&](uint32_t wd, uint32_t cnt) -> int {
            const uint64_t p = (uint64_t)wd * cnt;
            edge = edge || (uint32_t)p < cnt;
            return (int)(p >> 32);
        };
        const bool targeted = (uint64_t)b0.x < con->thr_target;
        const int rdraw = ix(b0.y, (uint32_t)n);
        int R1 = targeted ? hot : rdraw;
        const bool dbl = (uint64_t)b0.z < con->thr_dbl;
        bool flip = (uint64_t)b0.w < con->thr_sign;
        if (!ONEZ) flip = flip || E.w == n;
        flip = flip && !dbl;
        const bool rowswap = GEN && E.move_set == 1 && !flip && !dbl;
        const int r2d = ix(dbl ? b3.y : b1.y, (uint32_t)(dbl ? n : n - 1));
        int R2 = dbl ? (b3.x < 0x80000000u ? R1 : r2d) : r2d + (r2d >= R1 ? 1 : 0);
        if (flip || rowswap) R2 = R1;
        int C1, C2, p1 = 0, p2 = 0;
        bool bad;
        if constexpr (ONEZ) {
            // the row's only zero is its minority entry
            const int z1 = (int)lds8(E.mino + (uint32_t)R1), z2 = (int)lds8(E.mino + (uint32_t)R2);
            int f1 = ix(dbl ? b2.w : b1.x, (uint32_t)n), f2 = ix(b3.z, (uint32_t)n);
            f1 += f1 == z1 ? 1 : 0;
            f2 += f2 == z2 ? 1 : 0;
            if (f1 >= n) f1 = 0;
            if (f2 >= n) f2 = 0;
            const bool sw = !dbl && !flip;
            C1 = sw ? z2 : f1;
            C2 = sw ? z1 : dbl ? f2 : f1;
            bad = flip ? false : (R2 == R1 || sw) && C1 == C2;
        } else {
            auto fcol = [&](uint32_t wd, int row) -> int {
                const int i = ix(wd, (uint32_t)(sparse ? m : n));
                return sparse ? (int)lds8(E.mino + (uint32_t)(row * m + i)) : mask_first<WPL>(slot, row, i, n);
            };
            const int f1 = fcol(dbl ? b2.w : b1.x, R1);
            const int f2 = fcol(b3.z, R2);
            p1 = ix(b1.z, (uint32_t)m);
            p2 = ix(b1.w, (uint32_t)m);
            const int q1 = (int)lds8(E.mino + (uint32_t)(R1 * m + p1)), q2 = (int)lds8(E.mino + (uint32_t)(R2 * m + p2));
            const uint32_t e1 = lds8(wbase + (uint32_t)q2 * st + (uint32_t)R1);
            const uint32_t e2 = lds8(wbase + (uint32_t)q1 * st + (uint32_t)R2);
            if (dbl) {
                C1 = f1;
                C2 = f2;
                bad = R2 == R1 && C1 == C2;
            } else if (flip) {
                C1 = C2 = f1;
                bad = false;
            } else {
                C1 = sparse ? q1 : q2;
                C2 = sparse ? q2 : q1;
                bad = sparse ? e1 != 1u || e2 != 1u : e1 == 1u || e2 == 1u;
            }
        }
        bool s1 = (uint64_t)b2.x < con->thr_swsign, s2 = (uint64_t)b2.y < con->thr_swsign;
        int kind = dbl ? 2 : flip ? 0 : 1;
        if (rowswap) {
            kind = 3;
            bad = false;
        }
        const bool need = act && (bad || edge);
        if (__any_sync(gm, need)) {
            const uint2 x = propose_exact<WPL, GW>(need, slot, cw, E.mino, st, n, E.w, m, sparse, hot, c, it, E.stream, E.k0,
                                                   E.k1);
            if (need) {
                R1 = (int)(x.x & 255u);
                if (kind != 3) {
                    R2 = (int)((x.x >> 8) & 255u);
                    C1 = (int)((x.x >> 16) & 255u);
                    C2 = (int)(x.x >> 24);
                    kind = (int)(x.y & 3u);
                    p1 = (int)((x.y >> 8) & 255u);
                    p2 = (int)((x.y >> 16) & 255u);
                    s1 = (x.y >> 24) & 1u;
                    s2 = (x.y >> 25) & 1u;
                }
            }
        }

        if (GEN && kind == 3) {
            // the within-row swap: a nonzero of the row moves to one of its zeros
            const uint32_t dsl = cand_slot(c, 1);
            const int pos = (int)draw_index(sparse ? b1.y : b1.z, (uint32_t)m, dsl, it, E.stream, E.k0, E.k1, sparse ? 1 : 2);
            const int start = (int)draw_index(sparse ? b1.z : b1.y, (uint32_t)n, dsl, it, E.stream, E.k0, E.k1, sparse ? 2 : 1);
            const int q = (int)lds8(E.mino + (uint32_t)(R1 * m + pos));
            p1 = pos;
            R2 = R1;
            C1 = sparse ? q : mask_first<WPL>(slot, R1, start, n);
            C2 = sparse ? mask_first<WPL, true>(slot, R1, start, n) : q;
            s1 = b1.w < 0x80000000u;
        }

        // E: coefficients, then the new values of the lane's rows
        const uint32_t w1 = wbase + (uint32_t)C1 * st, w2 = wbase + (uint32_t)C2 * st;
        const int e11 = (int)lds8(w1 + (uint32_t)R1) - 1, e22 = (int)lds8(w2 + (uint32_t)R2) - 1;
        const int e21 = (int)lds8(w1 + (uint32_t)R2) - 1, e12 = (int)lds8(w2 + (uint32_t)R1) - 1;
        const bool two = R2 != R1;
        int a1 = kind == 1 || (GEN && kind == 3) ? -e11 : -2 * e11;
        int b1c = 0, a2 = 0, b2c = 0, pk = 0;
        if (kind == 1) {
            b1c = s1 ? -e11 : e11;
            a2 = s2 ? -e22 : e22;
            b2c = -e22;
        } else if (kind == 2) {
            if (two) {
                b2c = -2 * e22;
                // double flip over two rows (xweigh_cuda.cu:564-583)
                pk = a1 * e21 + b2c * e12 + (C1 == C2 ? a1 * b2c : 0);
            } else {
                b1c = -2 * e22;
            }
        } else if (GEN && kind == 3) {
            b1c = s1 ? 1 : -1;
        }
        uint32_t x[WPL], y[WPL], g1[WPL], g2[WPL];
        load_words<WPL>(w1 + E.loff, x);
        load_words<WPL>(w2 + E.loff, y);
        load_words<WPL>(E.g + (uint32_t)R1 * st + E.loff, g1);
        load_words<WPL>(E.g + (uint32_t)R2 * st + E.loff, g2);
        const uint32_t rs1 = lds32(slot + Slot<WPL>::res + 4u * (uint32_t)R1);
        const uint32_t rs2 = lds32(slot + Slot<WPL>::res + 4u * (uint32_t)R2);
        const uint32_t kk1 = (uint32_t)(-(a1 + b1c)) * 0x01010101u, kk2 = (uint32_t)(-(a2 + b2c)) * 0x01010101u;
        int acc = 0, pr = 0;
#pragma unroll
        for (int j = 0; j < WPL; ++j) {
            // columns R1 and R2 of the changed rows are left out (the entry
            // of a double flip over two rows apart): their W reads as zero
            const int widx = E.l * WPL + j;
            const uint32_t m1 = (R1 >> 2) == widx ? 0xffu << ((R1 & 3) * 8) : 0u;
            const uint32_t m2 = (R2 >> 2) == widx ? 0xffu << ((R2 & 3) * 8) : 0u;
            const uint32_t mm = m1 | m2;
            const uint32_t xx = (x[j] & ~mm) | (0x01010101u & mm), yy = (y[j] & ~mm) | (0x01010101u & mm);
            uint32_t n1 = g1[j] + kk1 + (uint32_t)a1 * xx + (uint32_t)b1c * yy;
            const uint32_t n2 = g2[j] + kk2 + (uint32_t)a2 * xx + (uint32_t)b2c * yy;
            if ((R2 >> 2) == widx) n1 += (uint32_t)pk << ((R2 & 3) * 8);
            const uint32_t v1 = __vabsdiffu4(n1, 0x80808080u), v2 = __vabsdiffu4(n2, 0x80808080u);
            const uint32_t z1 = (v1 + 0x7f7f7f7fu) & 0x80808080u, z2 = (v2 + 0x7f7f7f7fu) & 0x80808080u;
            uint32_t t = (uint32_t)acc;
            t = __dp4a(v1, 0x01010101u, t);
            t = __dp4a(v2, 0x01010101u, t);
            t = __dp4a(z1, 0x20202020u, t);   // 128 * 32: 4096 a conflict
            t = __dp4a(z2, 0x20202020u, t);
            acc = (int)t;
            if (GEN) {
                if (E.obj_kind == 1) {
                    const int d1 = (int)(n1 ^ 0x80808080u), d2 = (int)(n2 ^ 0x80808080u);
                    const int o1 = (int)(g1[j] ^ 0x80808080u), o2 = (int)(g2[j] ^ 0x80808080u);
                    pr = __dp4a(d1, d1, pr) + __dp4a(d2, d2, 0) - __dp4a(o1, o1, 0) - __dp4a(o2, o2, 0);
                } else if (E.obj_kind == 2) {
                    // 128 is even: the biased byte has the entry's parity
                    pr += __popc((n1 & 0x01010101u) | ((n2 & 0x01010101u) << 1)) -
                          __popc((g1[j] & 0x01010101u) | ((g2[j] & 0x01010101u) << 1));
                }
            }
        }
        if (!E.lact) {
            acc = 0;
            pr = 0;
        }
        if (E.l == 0) {
            const int r1 = (int)(rs1 & ((1u << kConfShift) - 1u)) + (int)((rs1 >> kConfShift) << 12);
            const int r2 = (int)(rs2 & ((1u << kConfShift) - 1u)) + (int)((rs2 >> kConfShift) << 12);
            acc -= r1 + r2;
        }
#pragma unroll
        for (int d = 1; d < LPC; d <<= 1) acc += __shfl_xor_sync(gm, acc, d);
        if (GEN && E.obj_kind != 0) {
#pragma unroll
            for (int d = 1; d < LPC; d <<= 1) pr += __shfl_xor_sync(gm, pr, d);
        }
        const int dc = (acc + 2048) >> 12;
        const int ds = acc - dc * 4096;
        cand_l += act ? 1u : 0u;
        two_l += act && two ? 1u : 0u;

        // the first best candidate: least (objective, score, conflicts, index)
        uint32_t ka, A, B = 0;
        if (!GEN || E.obj_kind == 0) {
            ka = ((uint32_t)(ds + 2048) << 14) | ((uint32_t)(dc + 256) << 5) | (uint32_t)c;
            A = __reduce_min_sync(gm, act ? ka : 0xffffffffu);
        } else {
            ka = ((uint32_t)(pr + (1 << 19)) << 12) | (uint32_t)(ds + 2048);
            A = __reduce_min_sync(gm, act ? ka : 0xffffffffu);
            B = __reduce_min_sync(gm, act && ka == A ? ((uint32_t)(dc + 256) << 5) | (uint32_t)c : 0xffffffffu);
        }
        if (A < bestA || (GEN && A == bestA && B < bestB)) {
            bestA = A;
            bestB = B;
            const uint32_t sup = kind == 1 ? 3u << 24 : GEN && kind == 3 ? 1u << 24 : 0u;
            P.mv.rc = (uint32_t)R1 | ((uint32_t)R2 << 8) | ((uint32_t)C1 << 16) | ((uint32_t)C2 << 24);
            P.mv.cf = (uint32_t)(a1 & 255) | ((uint32_t)(b1c & 255) << 8) | ((uint32_t)(a2 & 255) << 16) |
                      ((uint32_t)b2c << 24);
            P.mv.ax = (uint32_t)(pk & 255) | ((uint32_t)p1 << 8) | ((uint32_t)p2 << 16) | sup;
            const uint32_t k = !GEN || E.obj_kind == 0 ? A : B;
            // the group's first lane of the winning candidate, within the warp
            P.src = (int)(threadIdx.x & 31u & ~(uint32_t)(GW - 1)) + (int)((k & 3u)) * LPC;
            P.dc = (int)((k >> 5) & 511u) - 256;
            if (!GEN || E.obj_kind == 0) {
                P.ds = (int)(A >> 14) - 2048;
                P.prim = P.ds;
            } else {
                P.ds = (int)(A & 4095u) - 2048;
                P.prim = (int)(A >> 12) - (1 << 19);
            }
            if (count > 4) {
                P.mv.rc = __shfl_sync(gm, P.mv.rc, P.src);
                P.mv.cf = __shfl_sync(gm, P.mv.cf, P.src);
                P.mv.ax = __shfl_sync(gm, P.mv.ax, P.src);
            }
        }
        c0 += 4;
        if (c0 >= count) break;
        // the next four candidates' draws
        __syncwarp(gm);
        dbuf[lane] = draw_block(E.my_slot + 128u * (uint32_t)c0, it, E.stream, E.k0, E.k1);
        if constexpr (GW == 16) dbuf[lane + 16] = draw_block(E.my_slot2 + 128u * (uint32_t)c0, it, E.stream, E.k0, E.k1);
        __syncwarp(gm);
    }
    return P;
}

__device__ __forceinline__ int packed_abs(int v) {
    // |v| and [v != 0] as they count into a packed residual
    return iabs(v) + (v != 0 ? 1 << kConfShift : 0);
}

// Commits a move (commit_*, xweigh_cuda.cu:607-877): the one or two Gram
// rows and their mirrored columns, the packed residuals, W, the support
// masks and the minority lists.  Lane o owns rows o, o + GW, ...
template <int WPL, bool GEN, int GW, bool ONEZ>
__device__ __forceinline__ void commit(const Env& E, const Move& mv, int lane) {
    constexpr int OPL = WPL;
    const unsigned gm = group_mask<GW>();
    const int n = E.n, m = ONEZ ? 1 : E.m, sparse = ONEZ ? 0 : E.sparse;
    const uint32_t st = E.st, slot = E.slot, wbase = E.slot + Slot<WPL>::w;
    const int R1 = (int)(mv.rc & 255u), R2 = (int)((mv.rc >> 8) & 255u);
    const int C1 = (int)((mv.rc >> 16) & 255u), C2 = (int)(mv.rc >> 24);
    const int a1 = (int)(int8_t)(mv.cf & 255u), b1 = (int)(int8_t)((mv.cf >> 8) & 255u);
    const int a2 = (int)(int8_t)((mv.cf >> 16) & 255u), b2 = (int)(int8_t)(mv.cf >> 24);
    const int pk = (int)(int8_t)(mv.ax & 255u);
    const bool two = R2 != R1;
    const uint32_t w1 = wbase + (uint32_t)C1 * st, w2 = wbase + (uint32_t)C2 * st;
    const uint32_t g1 = E.g + (uint32_t)R1 * st, g2 = E.g + (uint32_t)R2 * st;
    int S1 = 0, S2 = 0;
#pragma unroll
    for (int k = 0; k < OPL; ++k) {
        const int o = lane + GW * k;
        if (o < n && o != R1) {
            const int x = (int)lds8(w1 + (uint32_t)o) - 1, y = (int)lds8(w2 + (uint32_t)o) - 1;
            const int o1 = (int)lds8(g1 + (uint32_t)o) - 128;
            const bool pair = two && o == R2;
            const int n1 = o1 + (pair ? pk : a1 * x + b1 * y);
            const int d1 = packed_abs(n1) - packed_abs(o1);
            xw_smem[g1 + (uint32_t)o] = (uint8_t)(n1 + 128);
            xw_smem[E.g + (uint32_t)o * st + (uint32_t)R1] = (uint8_t)(n1 + 128);
            S1 += d1;
            int d2 = 0;
            if (two) {
                if (pair) {
                    S2 += d1;
                } else {
                    const int o2 = (int)lds8(g2 + (uint32_t)o) - 128;
                    const int n2 = o2 + a2 * x + b2 * y;
                    d2 = packed_abs(n2) - packed_abs(o2);
                    xw_smem[g2 + (uint32_t)o] = (uint8_t)(n2 + 128);
                    xw_smem[E.g + (uint32_t)o * st + (uint32_t)R2] = (uint8_t)(n2 + 128);
                    S2 += d2;
                }
            }
            if (!pair) {
                int* r = reinterpret_cast<int*>(xw_smem + slot + Slot<WPL>::res) + o;
                *r += d1 + d2;
            }
        }
    }
    S1 = __reduce_add_sync(gm, S1);
    S2 = two ? __reduce_add_sync(gm, S2) : 0;
    __syncwarp(gm);
    // one changed entry of W per lane 0..3; rows R1 (lane 0) and R2 (lane
    // 1): residual, support mask and minority entry
    if (lane < 4) {
        const int cfc = (int)(int8_t)((mv.cf >> (8 * lane)) & 255u);
        if (cfc != 0) {
            const uint32_t a = ((lane & 1) ? w2 : w1) + (uint32_t)((lane & 2) ? R2 : R1);
            xw_smem[a] = (uint8_t)(lds8(a) + (uint32_t)cfc);
        }
        if (lane == 0 || (lane == 1 && two)) {
            const int R = lane ? R2 : R1;
            int* r = reinterpret_cast<int*>(xw_smem + slot + Slot<WPL>::res) + R;
            *r += lane ? S2 : S1;
            if ((mv.ax >> (24 + lane)) & 1u) {
                if constexpr (WPL == 1) {
                    uint32_t* mk = reinterpret_cast<uint32_t*>(xw_smem + slot + Slot<WPL>::mask) + R;
                    *mk ^= (1u << C1) ^ (1u << C2);
                } else {
                    uint64_t* mk = reinterpret_cast<uint64_t*>(xw_smem + slot + Slot<WPL>::mask) + (WPL / 2) * R;
                    mk[C1 >> 6] ^= 1ull << (C1 & 63);
                    mk[C2 >> 6] ^= 1ull << (C2 & 63);
                }
                // row R1 loses C1 and gains C2, row R2 the other way
                const int lost = lane ? C2 : C1, got = lane ? C1 : C2;
                const int p = (int)((mv.ax >> (8 + 8 * lane)) & 255u);
                xw_smem[E.mino + (uint32_t)(R * m + p)] = (uint8_t)(sparse ? got : lost);
            }
        }
    }
    __syncwarp(gm);
}

// tab[d-1] = ceil(exp(-d/T) * 2^32), computed with the same division and
// exponential as metropolis_accept, so that for a 32-bit draw u
//   u * 2^-32 < exp(-d/T)  <=>  u < tab[d-1]
// exactly (both sides scaled by 2^32 without rounding; u is an integer).
// Rebuilt whenever the replica's temperature changes.
template <int GW = 32>
__device__ __noinline__ void build_thresholds(uint64_t* tab, double T, int lane) {
    const double t = T > 1.0e-12 ? T : 1.0e-12;
    for (uint32_t d = lane + 1; d <= kThrTable; d += GW) {
        const double e = acceptance_exp(__ddiv_rn(-(double)d, t));
        tab[d - 1] = (uint64_t)ceil(__dmul_rn(e, 0x1p32));
    }
    __syncwarp(group_mask<GW>());
}

template <int GW = 32>
__device__ __forceinline__ void copy16(void* dst, const void* src, uint32_t bytes, int lane) {
    const uint32_t chunks = xw_pad16(bytes) / 16u;
    uint4* d = reinterpret_cast<uint4*>(dst);
    const uint4* s = reinterpret_cast<const uint4*>(src);
    for (uint32_t i = lane; i < chunks; i += GW) d[i] = s[i];
}

__device__ __forceinline__ uint64_t globaltimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// The replica's W as int8, column-major, into its record.
template <int WPL, int GW>
__device__ __noinline__ void save_w(int8_t* dst, uint32_t wbase, uint32_t st, int n, int lane) {
#pragma unroll 1
    for (int c = 0; c < n; ++c)
        for (int r = lane; r < n; r += GW) dst[(uint32_t)(c * n + r)] = (int8_t)((int)lds8(wbase + (uint32_t)c * st + (uint32_t)r) - 1);
}

// Scalar state of a loaded replica.
struct State {
    uint8_t* rec;
    RepHeader* H;
    XwJob* J;
    uint64_t it;
    int score, conflicts, best_s, best_c, msi, cool;
    int64_t obj_total;
    uint32_t accepted, accepted_rows;
    // the best W is the current one and its record is older: it is written
    // when an accepted move leaves it, or at the end
    bool dirty;
    // the copy that writes the record (a cluster's other CTAs keep an
    // identical copy in their own shared memory and write nothing)
    bool owner;
};

// Lane-invariant parts of the context, from the job and the slot.
template <int WPL, int GW, bool ONEZ>
__device__ __forceinline__ void make_env(Env& E, const XwJob* J, const RepHeader* H, uint32_t slot, uint32_t draws,
                                         int lane, int obj_kind) {
    constexpr int LPC = GW / 4;
    const int n = J->n;
    E.slot = slot;
    E.draws = draws;
    E.n = n;
    E.w = ONEZ ? n - 1 : J->w;
    E.m = ONEZ ? 1 : J->m;
    E.sparse = ONEZ ? 0 : J->sparse;
    E.st = packed_stride(n, WPL);
    const uint32_t mat = xw_pad16((uint32_t)n * E.st);
    E.g = slot + Slot<WPL>::w + mat;
    E.mino = E.g + mat;
    E.k0 = J->key0;
    E.k1 = J->key1;
    E.stream = H->stream;
    E.cs = J->candidate_samples;
    E.ts = J->target_samples;
    E.bpc = 4 + (E.ts <= 4 ? 1 : 2);   // cached blocks per candidate
    E.move_set = J->move_set;
    E.obj_kind = obj_kind;
    E.l = lane & (LPC - 1);
    E.grp = lane / LPC;
    E.lact = 4 * WPL * E.l < n;
    E.loff = E.lact ? (uint32_t)(4 * WPL * E.l) : 0u;
    auto slot_of = [&](int q) -> uint32_t {
        if (q == 0) return 0u;
        const int c = (q - 1) / E.bpc;
        return cand_slot(c, (q - 1) - c * E.bpc);
    };
    E.my_slot = slot_of(lane);
    E.my_slot2 = GW == 16 ? slot_of(lane + 16) : 0u;
}

// Loads replica `rid` into the slot: W and the minority lists; the masks,
// the Gram matrix (by popcounts of support and sign masks) and the
// residuals are rebuilt from W and checked against the header.  False when
// the replica does not run (job done or solved, budget spent, or a failed
// self-check, which flags the header).  The group's lanes call it.
// `owner` false: a copy that writes nothing to the record; it also skips
// the exits on the job's done and solved flags, which other kernels may set
// while it loads (its owner decides whether the replica runs).
template <int WPL, bool GEN, int GW, bool ONEZ>
__device__ __forceinline__ bool load_replica(const AnnealArgs& a, uint32_t rid, uint32_t slot, uint32_t draws, int lane,
                                             uint64_t& iters, Env& E, State& S, bool owner) {
    constexpr int OPL = WPL;   // rows o, o + GW, ... of a lane: GW * OPL >= n
    const unsigned gm = group_mask<GW>();
    uint8_t* rec = a.arena + a.rec_off[rid];
    RepHeader* H = reinterpret_cast<RepHeader*>(rec);
    XwJob* J = a.jobs + H->job;
    S.rec = rec;
    S.H = H;
    S.J = J;
    S.owner = owner;
    if (owner && *(volatile int32_t*)&J->done) return false;
    if (owner && a.stop_on_solve == 1 && *(volatile int32_t*)&J->solved) return false;
    const int obj_kind = GEN ? H->obj_kind : 0;
    if ((ONEZ && (J->m != 1 || J->sparse != 0)) || (!GEN && (H->obj_kind != 0 || J->move_set != 0))) {
        // a launch of a specialised kernel met a replica it does not cover
        if (lane == 0) H->err |= XW_ERR_KERNEL;
        return false;
    }
    make_env<WPL, GW, ONEZ>(E, J, H, slot, draws, lane, obj_kind);
    const int n = E.n, w = E.w, m = E.m, sparse = E.sparse;
    S.it = H->it;
    if (J->budget_iters) {
        if (S.it >= J->budget_iters) return false;
        if (iters > J->budget_iters - S.it) iters = J->budget_iters - S.it;
    }
    const uint32_t status0 = H->status;
    const uint32_t st = E.st, wbase = slot + Slot<WPL>::w;

    // W as biased bytes, the pad rows zero (biased 1); support and sign
    // masks of the lane's rows
    uint32_t sup[OPL][WPL], neg[OPL][WPL];
#pragma unroll
    for (int k = 0; k < OPL; ++k)
#pragma unroll
        for (int q = 0; q < WPL; ++q) sup[k][q] = neg[k][q] = 0;
    int bad = 0;
    const int8_t* gw = reinterpret_cast<const int8_t*>(rec + J->off_w);
#pragma unroll
    for (int q = 0; q < WPL; ++q) {
#pragma unroll 1
        for (int c = 32 * q; c < n && c < 32 * q + 32; ++c) {
#pragma unroll
            for (int k = 0; k < OPL; ++k) {
                const int o = lane + GW * k;
                int v = 0;
                if (o < n) {
                    v = gw[(uint32_t)(c * n + o)];
                    if (v < -1 || v > 1) bad = 1;
                    if (v) sup[k][q] |= 1u << (c & 31);
                    if (v < 0) neg[k][q] |= 1u << (c & 31);
                }
                if ((uint32_t)o < st) xw_smem[wbase + (uint32_t)c * st + (uint32_t)o] = (uint8_t)(v + 1);
            }
            // the stride's pad beyond the lanes' rows
            for (uint32_t o = (uint32_t)(lane + GW * OPL); o < st; o += GW) xw_smem[wbase + (uint32_t)c * st + o] = 1;
        }
    }
    // an empty list still reads as column 0
    if (m == 0 && lane == 0) xw_smem[E.mino] = 0;
    if (m > 0 && (status0 & XW_STATUS_INIT)) {
        const uint8_t* gm8 = rec + J->off_mino;
        for (uint32_t i = lane; i < (uint32_t)(n * m); i += GW) xw_smem[E.mino + i] = gm8[i];
    }
#pragma unroll
    for (int k = 0; k < OPL; ++k) {
        const int o = lane + GW * k;
        if (o < n) {
            int weight = 0;
#pragma unroll
            for (int q = 0; q < WPL; ++q) {
                *reinterpret_cast<uint32_t*>(xw_smem + slot + Slot<WPL>::mask + (uint32_t)(o * WPL + q) * 4u) = sup[k][q];
                weight += __popc(sup[k][q]);
            }
            if (weight != w) bad = 1;
            if (m > 0 && !(status0 & XW_STATUS_INIT) && weight == w) {
                // minority list in column order: the nonzeros of a sparse
                // row, the zeros of a dense one (m entries either way)
                int pos = 0;
#pragma unroll
                for (int q = 0; q < WPL; ++q) {
                    const int left = n - 32 * q;
                    const uint32_t valid = left >= 32 ? 0xffffffffu : left > 0 ? (1u << left) - 1u : 0u;
                    uint32_t x = (sparse ? sup[k][q] : ~sup[k][q]) & valid;
                    while (x) {
                        xw_smem[E.mino + (uint32_t)(o * m + pos)] = (uint8_t)(32 * q + __ffs((int)x) - 1);
                        x &= x - 1;
                        ++pos;
                    }
                }
            }
        }
    }
    if (__any_sync(gm, bad)) {
        if (lane == 0 && owner) H->err |= XW_ERR_MINORITY;
        return false;
    }
    __syncwarp(gm);
    int p_score = 0, p_conf = 0, p_par = 0;
    long long p_sq = 0;
#pragma unroll
    for (int k = 0; k < OPL; ++k) {
        int r_sum = 0;
        const int o = lane + GW * k;
#pragma unroll
        for (int kr = 0; kr < OPL; ++kr) {
#pragma unroll 1
            for (int lr = 0; lr < GW; ++lr) {
                const int r = lr + GW * kr;
                if (r >= n) break;
                int dot = 0;
#pragma unroll
                for (int q = 0; q < WPL; ++q) {
                    const uint32_t both = sup[k][q] & lds32(slot + Slot<WPL>::mask + (uint32_t)(r * WPL + q) * 4u);
                    const uint32_t ng = __shfl_sync(gm, neg[kr][q], lr, GW);
                    dot += __popc(both) - 2 * __popc(both & (neg[k][q] ^ ng));
                }
                if (o < n) {
                    if (r == o) dot = 0;   // the diagonal is kept at 0
                    xw_smem[E.g + (uint32_t)r * st + (uint32_t)o] = (uint8_t)(dot + 128);
                    r_sum += packed_abs(dot);
                    p_sq += (long long)(dot * dot);
                    p_par += dot & 1;
                } else if ((uint32_t)o < st) {
                    xw_smem[E.g + (uint32_t)r * st + (uint32_t)o] = 128;
                }
                if (k == OPL - 1)
                    for (uint32_t p = (uint32_t)(lane + GW * OPL); p < st; p += GW) xw_smem[E.g + (uint32_t)r * st + p] = 128;
            }
        }
        if (o < n) {
            reinterpret_cast<int*>(xw_smem + slot + Slot<WPL>::res)[o] = r_sum;
            p_score += r_sum & ((1 << kConfShift) - 1);
            p_conf += r_sum >> kConfShift;
        }
    }
    const int score0 = __reduce_add_sync(gm, p_score) / 2;
    const int conf0 = __reduce_add_sync(gm, p_conf) / 2;
#pragma unroll
    for (int off = GW / 2; off > 0; off >>= 1) p_sq += __shfl_xor_sync(gm, p_sq, off, GW);
    const long long sq0 = p_sq / 2;
    const int par0 = __reduce_add_sync(gm, p_par) / 2;
    __syncwarp(gm);

    const int64_t obj0 = obj_kind == 1 ? sq0 : obj_kind == 2 ? par0 : score0;
    if (status0 & XW_STATUS_INIT) {
        if (H->score != score0 || H->conflicts != conf0 || H->obj_total != obj0) {
            if (lane == 0 && owner) H->err |= XW_ERR_SCORE;
            return false;
        }
        S.best_s = H->best_score;
        S.best_c = H->best_conflicts;
        S.msi = H->msi;
        S.cool = H->cool_ctr;
        S.accepted = H->accepted;
        S.accepted_rows = H->accepted_rows;
        S.dirty = false;
    } else {
        S.best_s = score0;
        S.best_c = conf0;
        S.msi = 0;
        S.cool = 0;
        S.accepted = 0;
        S.accepted_rows = 0;
        S.dirty = true;
    }
    S.score = score0;
    S.conflicts = conf0;
    S.obj_total = obj0;
    if (lane == 0) {
        Con c;
        c.thr_target = J->thr_target;
        c.thr_dbl = GEN && J->move_set == 1 ? 0 : J->thr_double;
        c.thr_sign = J->thr_sign;
        c.thr_swsign = J->thr_swsign;
        c.thr_greedy = J->thr_greedy;
        c.T = H->temperature;
        *reinterpret_cast<Con*>(xw_smem + slot + Slot<WPL>::con) = c;
    }
    __syncwarp(gm);
    build_thresholds<GW>(reinterpret_cast<uint64_t*>(xw_smem + slot + Slot<WPL>::thr), H->temperature, lane);
    return true;
}

// Writes the replica's W, minority lists and scalar state back to its
// record; `calls` moves were made since it was loaded, with `evals`
// candidates evaluated, `evals2` of them changing two rows.
template <int WPL, int GW>
__device__ __forceinline__ void store_replica(const Env& E, State& S, uint64_t calls, uint64_t evals, uint32_t evals2,
                                              int lane) {
    const unsigned gm = group_mask<GW>();
    __syncwarp(gm);
    if (S.dirty) save_w<WPL, GW>(reinterpret_cast<int8_t*>(S.rec + S.J->off_best), E.slot + Slot<WPL>::w, E.st, E.n, lane);
    save_w<WPL, GW>(reinterpret_cast<int8_t*>(S.rec + S.J->off_w), E.slot + Slot<WPL>::w, E.st, E.n, lane);
    uint8_t* gmo = S.rec + S.J->off_mino;
    for (uint32_t i = lane; i < (uint32_t)(E.n * E.m); i += GW) gmo[i] = xw_smem[E.mino + i];
    if (lane == 0) {
        RepHeader* H = S.H;
        const bool init = H->status & XW_STATUS_INIT;
        H->it = S.it;
        H->moves = (init ? H->moves : 0) + calls;
        H->cand_evals = (init ? H->cand_evals : 0) + evals;
        H->accepted = S.accepted;
        H->accepted_rows = S.accepted_rows;
        H->two_row_evals = (init ? H->two_row_evals : 0) + evals2;
        H->score = S.score;
        H->conflicts = S.conflicts;
        H->best_score = S.best_s;
        H->best_conflicts = S.best_c;
        H->obj_total = S.obj_total;
        H->temperature = reinterpret_cast<const Con*>(xw_smem + E.slot + Slot<WPL>::con)->T;
        H->msi = S.msi;
        H->cool_ctr = S.cool;
        H->status = H->status | XW_STATUS_INIT | (S.best_s == 0 ? XW_STATUS_SOLVED : 0u);
    }
    __syncwarp(gm);
}

// The Metropolis test of a chosen move at the replica's temperature (xweigh_cuda.cu:1040-1060).
template <int WPL>
__device__ __forceinline__ bool accepts(const Env& E, const Pick& P) {
    if (P.prim <= 0) return true;
    if (P.prim <= (int)kThrTable) return (uint64_t)P.u < lds64(E.slot + Slot<WPL>::thr + 8u * (uint32_t)(P.prim - 1));
    return metropolis_accept(P.prim, reinterpret_cast<const Con*>(xw_smem + E.slot + Slot<WPL>::con)->T, P.u);
}

// One move call whose Metropolis outcome is `accept`: the commit, best
// tracking (and the job's solve flag), cooling and reheat
// (xweigh_cuda.cu:1087-1129).  S.it is the iteration's number.
template <int WPL, bool GEN, int GW, bool ONEZ>
__device__ __forceinline__ void apply(const Env& E, State& S, Pick& P, bool accept, int tempering, int mpc, int stuck,
                                      int lane) {
    const unsigned gm = group_mask<GW>();
    bool improved = false;
    if (accept) {
        const int ns = S.score + P.ds, nc = S.conflicts + P.dc;
        improved = ns < S.best_s || (ns == S.best_s && nc < S.best_c);
        if (S.dirty && !improved) {
            if (S.owner)
                save_w<WPL, GW>(reinterpret_cast<int8_t*>(S.rec + S.J->off_best), E.slot + Slot<WPL>::w, E.st, E.n, lane);
            S.dirty = false;
            __syncwarp(gm);
        }
        P.mv.rc = __shfl_sync(gm, P.mv.rc, P.src);
        P.mv.cf = __shfl_sync(gm, P.mv.cf, P.src);
        P.mv.ax = __shfl_sync(gm, P.mv.ax, P.src);
        commit<WPL, GEN, GW, ONEZ>(E, P.mv, lane);
        S.score = ns;
        S.conflicts = nc;
        S.obj_total += P.prim;
        ++S.accepted;
        S.accepted_rows += (P.mv.rc & 255u) != ((P.mv.rc >> 8) & 255u) ? 2u : 1u;
        if (improved) {
            S.best_s = ns;
            S.best_c = nc;
            S.dirty = true;
            if (ns == 0 && lane == 0 && S.owner) {
                RepHeader* H = S.H;
                XwJob* J = S.J;
                H->solve_it = S.it;
                H->solve_ns = globaltimer();
                if (atomicCAS(&J->solved, 0, 1) == 0) {
                    J->solved_replica = (int32_t)H->stream;
                    J->solved_it = S.it;
                    J->solve_ns = H->solve_ns;
                }
            }
        }
    }
    S.msi = improved ? 0 : S.msi + 1;
    if (!tempering) {
        ++S.cool;
        if (S.cool >= mpc || S.msi >= stuck) {
            Con* con = reinterpret_cast<Con*>(xw_smem + E.slot + Slot<WPL>::con);
            const double T0 = con->T, t_min = S.J->t_min;
            double T = T0;
            if (S.cool >= mpc) {
                S.cool = 0;
                T = __dmul_rn(T, S.J->cooling);
                if (T < t_min) T = t_min;
            }
            if (S.msi >= stuck) {
                S.msi = 0;
                T = __dmul_rn(S.H->reheat_temperature, S.J->reheat);
                if (T < t_min) T = t_min;
            }
            __syncwarp(gm);
            if (lane == 0) con->T = T;
            if (T != T0) build_thresholds<GW>(reinterpret_cast<uint64_t*>(xw_smem + E.slot + Slot<WPL>::thr), T, lane);
            __syncwarp(gm);
        }
    }
}

}  // namespace
}  // namespace xw
