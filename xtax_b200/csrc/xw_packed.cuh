// xw_packed.cuh -- one annealing iteration on packed rows, for orders up to
// 448: the device code shared by the one-warp replica loop (xw_replica.cuh),
// the latency mode (xw_spec.cuh) and the large orders' kernel
// (xw_anneal_wide.cu).
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
// What bounds it: instruction issue of dependent integer chains (W(26,25)
// ladder, 4096 replicas: issue slots 62% used, ALU pipe 55%, 395 warp
// instructions an iteration with load and store, 19.2 ms per 10^4 of them).
// Measured on B200 against a loop over candidates with one row per lane and
// a 32-bit Gram matrix (838 instructions, 44.7 ms): packed rows alone 30.5
// ms; runs of one-candidate iterations side by side and the constants and
// the state of accepted moves in shared memory instead of registers 26.9; no
// calls in the loop (a call keeps what lives across it in few registers: 80
// bytes of spills a thread) and round keys from shared memory 19.2.
// W(100,50), 592 replicas of 1000 iterations: 13.6 -> 5.1 ms (bytes let six
// warps share an SM instead of three; the lanes try a switch's attempts side
// by side), 3.7 with the journal of moves since the best W.
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
    if (wpl == 8) return ((uint32_t)n + 7u) & ~7u;
    if (wpl == 16) return 4u * (((uint32_t)n + 15u) >> 4);   // four nibble pairs to 16 rows
    const uint32_t q = 4u * (uint32_t)wpl;
    return ((((uint32_t)n + q - 1u) / q) | 1u) * q;
}

// Orders above 128 (WPL 8): G as biased halfwords (+32768), eight to a
// 16-byte chunk, an odd number of chunks to a row; 32 chunks (orders above
// 248, which leave no room for a pad) have theirs permuted by the row
// instead.
__host__ __device__ constexpr uint32_t wide_stride(int n) {
    const uint32_t k = ((uint32_t)n + 7u) / 8u;
    return (k == 32u ? k : k | 1u) * 16u;
}

__device__ __forceinline__ uint32_t wide_at(uint32_t g, uint32_t gst, int row, int chunk) {
    return g + (uint32_t)row * gst + ((uint32_t)(chunk ^ (gst == 512u ? row & 7 : 0)) << 4);
}

// Moves since the best W that are kept to be undone when it is written: a
// chain that improves every few moves writes it only when it ends (a save at
// each move that left the best took 3000 of 3900 instructions an iteration
// of W(256,255) from a random start, 1000 of 1750 of W(100,50)).
constexpr int kJournal = 32;

// A replica's constants and the state that changes with an accepted move
// or a temperature step, in the slot: every lane reads them by broadcast
// when it needs them, lane 0 writes.  Kept there they cost the iteration a
// few broadcast reads instead of the registers that set how many warps
// share an SM.
//
// Calls are counted in k from the start of the launch; msi (calls since the
// last improvement) and the cooling counter are k - mb and k - cb.
struct Con {
    uint4 coins;         // the four thresholds below, at most 2^32 - 1
    uint4 keys[5];       // Philox round keys, two rounds each
    uint32_t k0, k1, stream;
    int32_t cs;
    uint64_t thr_target, thr_dbl, thr_sign, thr_swsign;
    uint64_t it0;        // iteration number at k = 0
    uint64_t thr_greedy;
    int4 best;           // score, conflicts, best score, best conflicts
    int4 acc;            // objective total (64 bits), accepted moves, rows they changed
    double T;
    int32_t mb, cb;
    int32_t mpc, stuck;  // calls per cooling step, calls without improvement before a reheat
    int32_t fixed;       // tempering: the temperature is the rung's, which only an exchange changes
    int32_t k_end;       // iterations of this launch
    // moves accepted since the best W, all of them in the journal: the record
    // holds an older one.  -1: the record holds the best W.
    int32_t jn;
    // the copy that writes the record (a cluster's other CTAs keep an
    // identical copy in their own shared memory and write nothing)
    int32_t owner;
    uint32_t rid;
    int32_t halves;      // hybrid form: G is in halfwords
};

// The slot: fixed regions first, so that their offsets are constants.
template <int WPL>
struct Slot {
    static constexpr uint32_t draws = 0;                      // 24 Philox blocks, then the window
    static constexpr uint32_t win = 384;                      // acceptance draws of 32 iterations
    static constexpr uint32_t thr = 512;                      // Metropolis thresholds
    static constexpr uint32_t jrn = thr + 4u * kThrTable;     // journal
    static constexpr uint32_t con = jrn + 8u * kJournal;
    static constexpr uint32_t res = con + 240u;               // packed residuals, 4 bytes a row
    static constexpr uint32_t mask = res + 128u * WPL;        // support masks, 4*WPL bytes a row
    static constexpr uint32_t w = mask + (WPL >= 8 ? 0u : 128u * WPL * WPL);
};

static_assert(sizeof(Con) <= 240, "replica constants fit their region");

__host__ __device__ constexpr uint32_t packed_slot_bytes(int n, int m, int wpl) {
    const uint32_t fixed = 512u + 4u * kThrTable + 8u * (uint32_t)kJournal + 240u + 128u * (uint32_t)wpl +
                           (wpl == 8 ? 0u : 128u * (uint32_t)(wpl * wpl));
    const uint32_t mat = xw_pad16((uint32_t)n * packed_stride(n, wpl));
    const uint32_t gram = wpl == 8 ? (uint32_t)n * wide_stride(n) : mat;
    // the minority lists' pad covers the read of an empty list
    return fixed + mat + gram + xw_pad16((uint32_t)(n * m) + 1u);
}

// The hybrid form of the large-order kernel (WPL 16, orders up to 448): W in
// the slot as nibble pairs, a byte to four rows of a column (low nibble
// support, high nibble sign), G in the replica's arena in HBM, rows of
// 16-byte chunks; the minority lists (16 bits) in the slot when they take at
// most kHybridMino bytes, else in the record.  G is kept as biased bytes
// while its entries stay within kByteMax (a move changes one by at most 4;
// entries of random rows have a standard deviation of sqrt(w)), and goes
// over to biased halfwords for good when a row that is read holds a larger
// one: half the bytes keep the Gram matrices of twice the replicas in L2.
// Tables at the start of the CTA's shared memory turn a nibble pair into
// four byte entries of W (one word) or four halfwords (two).
constexpr int kHybridMaxOrder = 448;
constexpr uint32_t kHybridMino = 8192;
constexpr uint32_t kNibbleTable = 2048 + 1024;
constexpr int kByteMax = 123;

// A candidate's two deltas travel in one word, score change + 4096 x conflict
// change: a move changes at most 2n entries of G by at most 2 each (or n by
// 4), so the score change of any order here stays below 2048.
static_assert(4 * kHybridMaxOrder < 2048, "score changes fit half of 4096");

__host__ __device__ constexpr uint32_t hybrid_slot_bytes(int n, int m) {
    const uint32_t mb = (uint32_t)n * (uint32_t)m * 2u;
    return 512u + 4u * kThrTable + 8u * (uint32_t)kJournal + 240u + xw_pad16(4u * (uint32_t)n) +
           xw_pad16((uint32_t)n * packed_stride(n, 16)) + (mb <= kHybridMino ? xw_pad16(mb + 2u) : 0u);
}

__host__ __device__ constexpr uint32_t hybrid_gram_stride(int n) { return (((uint32_t)n + 7u) >> 3) * 16u; }
__host__ __device__ constexpr uint32_t hybrid_byte_stride(int n) { return ((uint32_t)n + 15u) & ~15u; }

__host__ __device__ constexpr uint32_t hybrid_row_stride(int n) { return (((uint32_t)n + 63u) >> 6) * 32u; }

// The arena of a replica in that form: packed residuals, the rows of W as
// signed nibbles (used while G is built; in their place then a word that says
// whether G is in halfwords and, 16 bytes on, the slot's W for the next
// launch), G (room for halfwords).
struct HybridArena {
    uint64_t off_rows, off_g, bytes;
};

__host__ __device__ constexpr HybridArena hybrid_arena(int n) {
    HybridArena A{};
    A.off_rows = (4u * (uint64_t)n + 15u) & ~uint64_t(15);
    A.off_g = A.off_rows + (uint64_t)n * hybrid_row_stride(n);
    A.bytes = A.off_g + (uint64_t)n * hybrid_gram_stride(n);
    return A;
}

// bytes of the slot's W; it fits the place of the rows
__host__ __device__ constexpr uint32_t hybrid_w_bytes(int n) { return xw_pad16((uint32_t)n * packed_stride(n, 16)); }

constexpr bool hybrid_w_fits() {
    for (int n = 1; n <= kHybridMaxOrder; ++n)
        if (16u + hybrid_w_bytes(n) > (uint32_t)n * hybrid_row_stride(n)) return false;
    return true;
}
static_assert(hybrid_w_fits(), "the slot's W fits the arena's rows");

// Loop-invariant context of a lane of a replica's group.
struct Env {
    uint32_t slot;       // the replica's slot in xw_smem
    uint32_t draws;      // this group's draw buffer
    uint32_t cw;         // the cached draw blocks of this lane's candidate
    uint32_t g, mino;    // byte offsets of G and the minority lists
    uint32_t st;         // bytes from a column of W (and, up to order 128, a row of G) to the next
    uint32_t gst;        // the same of G above order 128
    uint8_t* gp;         // hybrid form: G in the arena, the minority lists
    uint16_t* mp;
    int n, m, sparse;
    // every move but the double flips is a sign flip: w = n, or (kernels with
    // row swaps) a coin of 2^32
    int flips;
    int ts, bpc, move_set, obj_kind;
    uint32_t dq[2];      // draw blocks this lane computes: candidate (or iteration) << 16 | 1 + block
};

// Entry (r, c) of W plus one.
template <int WPL>
__device__ __forceinline__ uint32_t w_at(uint32_t wbase, uint32_t st, int r, int c) {
    if constexpr (WPL == 16) {
        const uint32_t b = lds8(wbase + (uint32_t)c * st + ((uint32_t)r >> 2)) >> (r & 3);
        return 1u + (b & 1u) - 2u * ((b >> 4) & 1u);
    } else {
        return lds8(wbase + (uint32_t)c * st + (uint32_t)r);
    }
}

template <int WPL>
__device__ __forceinline__ int mino_at(const Env& E, int i) {
    if constexpr (WPL == 16) return E.mp[i];
    else return (int)lds8(E.mino + (uint32_t)i);
}

template <int WPL>
__device__ __forceinline__ Con* con_of(uint32_t slot) {
    return reinterpret_cast<Con*>(xw_smem + slot + Slot<WPL>::con);
}

// ---- proposals --------------------------------------------------------

__device__ __forceinline__ int first_from(uint32_t m, int start) {
    const uint32_t hi = m & (0xffffffffu << start);
    return __ffs((int)(hi ? hi : m)) - 1;
}

__device__ __forceinline__ int first_from(uint64_t m, int start) {
    const uint64_t hi = m & (~0ull << start);
    return __ffsll((long long)(hi ? hi : m)) - 1;
}

// W's offset: a slot of the hybrid form has its residuals just before.
template <int WPL>
__device__ __forceinline__ uint32_t wbase_of(uint32_t slot, int n) {
    return slot + (WPL == 16 ? Slot<WPL>::res + xw_pad16(4u * (uint32_t)n) : Slot<WPL>::w);
}

// First set bit at or after `start`, cyclically, of row `row`'s support
// mask (COMPL: of its complement below n).
template <int WPL, bool COMPL = false>
__device__ __forceinline__ int mask_first(uint32_t slot, int row, int start, int n) {
    const uint32_t a = slot + Slot<WPL>::mask + (uint32_t)row * (4u * WPL);
    if constexpr (WPL >= 8) {
        // no masks: the columns in turn (at most n / w of them, or n / (n - w)
        // zeros, on average, and only the fuller kind is searched this way)
        const uint32_t w = wbase_of<WPL>(slot, n), st = packed_stride(n, WPL);
        int c = start;
        while ((w_at<WPL>(w, st, row, c) == 1u) != COMPL) c = c + 1 == n ? 0 : c + 1;
        return c;
    } else if constexpr (WPL == 1) {
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

// The same in a row whose only zero is column z.
__device__ __forceinline__ int after_zero(int start, int z, int n) {
    const int c = start + (start == z ? 1 : 0);
    return c >= n ? 0 : c;
}

// A draw word outside the cached blocks (tournaments past 8 samples).
__device__ __forceinline__ uint32_t slow_word(uint32_t slot, uint64_t it, uint32_t stream, uint32_t k0, uint32_t k1,
                                           int j) {
    return pick(draw_block(slot, it, stream, k0, k1), j);
}

// Column of a sign flip in `row` from draw word `wd` (slot, word j of block
// b), propose_sign_flip (xweigh_cuda.cu:302-325): a minority pick for a
// sparse row, else the first nonzero at or after a random column.
template <int WPL, bool ONEZ>
__device__ __forceinline__ int flip_col_exact(const Env& E, uint32_t wd, uint32_t dslot, uint64_t it, uint32_t stream,
                                              uint32_t k0, uint32_t k1, int j, int row) {
    const int n = E.n;
    if constexpr (ONEZ)
        return after_zero((int)draw_index(wd, (uint32_t)n, dslot, it, stream, k0, k1, j), mino_at<WPL>(E, row), n);
    if (E.sparse && E.m > 0)
        return mino_at<WPL>(E, row * E.m + (int)draw_index(wd, (uint32_t)E.m, dslot, it, stream, k0, k1, j));
    return mask_first<WPL>(E.slot, row, (int)draw_index(wd, (uint32_t)n, dslot, it, stream, k0, k1, j), n);
}

// The row of a group's largest tournament key; `mine`: the row behind the
// lane's own (a key has room for its low eight bits, distinct by sample).
template <int WPL, int LPC>
__device__ __forceinline__ int best_row(uint32_t key, uint32_t mine, unsigned gm) {
    uint32_t top = key;
#pragma unroll
    for (int d = 1; d < LPC; d <<= 1) top = max(top, __shfl_xor_sync(gm, top, d));
    if constexpr (WPL < 16) return (int)(top & 255u);
    const int wl = (int)(threadIdx.x & 31u), base = wl & ~(LPC - 1);
    const uint32_t at = (__ballot_sync(gm, key == top) >> base) & ((1u << LPC) - 1u);
    return (int)__shfl_sync(gm, mine, base + __ffs((int)at) - 1);
}

// Hot-row tournament of candidate `c` (hot_row, xweigh_cuda.cu:291-300),
// the samples spread over the group's lanes: the first sample with the
// largest residual.
template <int WPL, int GW>
__device__ __forceinline__ int tournament(uint32_t slot, uint32_t cw, int n, int ts, int c, uint64_t it, int l,
                                          unsigned gm) {
    constexpr int LPC = GW / 4;
    const Con* con = con_of<WPL>(slot);
    uint32_t key = 0, mine = 0;
#pragma unroll 1
    for (int s = l; s < ts; s += LPC) {
        const uint32_t ds = cand_slot(c, 4 + (s >> 2));
        const uint32_t wd = s < 8 ? lds32(cw + 64u + 4u * (uint32_t)s)
                                  : slow_word(ds, it, con->stream, con->k0, con->k1, s & 3);
        const uint32_t r = draw_index(wd, (uint32_t)n, ds, it, con->stream, con->k0, con->k1, s & 3);
        const uint32_t k = (lds32(slot + Slot<WPL>::res + 4u * r) << 14) | ((uint32_t)(63 - s) << 8) | (r & 255u);
        if (k > key) {
            key = k;
            mine = r;
        }
    }
    return best_row<WPL, LPC>(key, mine, gm);
}

// The whole proposal of candidate `c` with exact index draws and every
// further attempt, propose_move (xweigh_cuda.cu:327-447): taken by the
// groups whose first attempt is not legal (a second flip that repeats the
// first, a switch whose 2x2 is not legal) or whose draws met Lemire's
// rejection zone.  Attempts are independent given their counters, so the
// group's lanes try several at once and the first legal one is taken; in
// order this is one attempt after the other, each with its own Philox
// blocks.  `need`: this lane's group wants a proposal (the other lanes take
// part in the collectives only); `from`: the first attempt to try (1 when
// attempt 0 is known to fail).  Returns
// {R1 | R2<<16, C1 | C2<<16, p1 | p2<<16, kind | s1<<2 | s2<<3}.
template <int WPL, int GW, bool ONEZ>
__device__ __forceinline__ uint4 propose_exact(const Env& E, bool need, int from, int hot, int c, uint64_t it, int l) {
    constexpr int LPC = GW / 4;
    const unsigned gm = group_mask<GW>();
    const int wl = threadIdx.x & 31, base = wl - l;
    const uint32_t slot = E.slot, cw = E.cw, st = E.st, wbase = wbase_of<WPL>(E.slot, E.n);
    const int n = E.n, m = ONEZ ? 1 : E.m, sparse = ONEZ ? 0 : E.sparse;
    const Con* con = con_of<WPL>(slot);
    const uint32_t k0 = con->k0, k1 = con->k1, stream = con->stream;
    auto ix = [&](uint32_t wd, uint32_t count, int b, int j) -> int {
        return (int)draw_index(wd, count, cand_slot(c, b), it, stream, k0, k1, j);
    };
    auto fcol = [&](uint32_t wd, int b, int j, int row) -> int {
        return flip_col_exact<WPL, ONEZ>(E, wd, cand_slot(c, b), it, stream, k0, k1, j, row);
    };
    int row = 0, r2 = 0, c1 = 0, c2 = 0, p1 = 0, p2 = 0, kind = -1;
    bool s1 = false, s2 = false, dbl = false, flip = false;
    if (need) {
        const uint4 b0 = lds128(cw);
        row = (uint64_t)b0.x < con->thr_target ? hot : ix(b0.y, (uint32_t)n, 0, 1);
        dbl = (uint64_t)b0.z < con->thr_dbl;
        flip = (!ONEZ && E.flips) || (uint64_t)b0.w < con->thr_sign;
    }
    // double flip (xweigh_cuda.cu:389-421): attempt 0 from block 3, attempt
    // a > 0 from block 19 + a, 16 in all
    bool pend = need && dbl;
    if (__any_sync(gm, pend)) {
        const int first = pend ? fcol(lds32(cw + 44u), 2, 3, row) : 0;
#pragma unroll 1
        for (int a0 = from; a0 < 16; a0 += LPC) {
            const int a = a0 + l;
            int rr = 0, cc = 0;
            bool ok = false;
            if (pend && a < 16) {
                const int b = a == 0 ? 3 : 19 + a;
                const uint4 d = a == 0 ? lds128(cw + 48) : draw_block(cand_slot(c, b), it, stream, k0, k1);
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
        c1 = c2 = fcol(lds32(cw + 16u), 1, 0, row);
    }
    // support switch (xweigh_cuda.cu:327-387): attempt 0 in blocks 1 and 2,
    // attempt a > 0 in blocks 36 + 2(a-1) and the next, 24 in all.  The
    // lower half of the lanes takes an attempt each, the upper half computes
    // the second blocks (a double flip that failed has not tried attempt 0).
    pend = need && kind < 0 && m > 0 && n > 1;
    if (__any_sync(gm, pend)) {
        constexpr int AT = LPC / 2;
        const bool second = l >= AT;
#pragma unroll 1
        for (int a0 = __any_sync(gm, pend && dbl) ? 0 : from; a0 < 24; a0 += AT) {
            const int a = a0 + (l & (AT - 1)), b = a == 0 ? 1 : 36 + 2 * (a - 1), o = a == 0 ? 1 : 0;
            int rr = 0, x1 = 0, pp = 0;
            uint4 d = make_uint4(0, 0, 0, 0);
            bool ok = false;
            if (pend && a < 24) {
                d = draw_block(cand_slot(c, b + (second ? 1 : 0)), it, stream, k0, k1);
                if (a == 0) {
                    const uint4 e = lds128(cw + 16), f = lds128(cw + 32);
                    d = second ? make_uint4(f.y, 0, 0, 0) : make_uint4(e.y, e.z, e.w, f.x);
                }
                if (!second) {
                    rr = ix(d.x, (uint32_t)(n - 1), b, o);
                    if (rr >= row) ++rr;
                    const int q = ix(d.y, (uint32_t)m, b, o + 1), qq = ix(d.z, (uint32_t)m, b, o + 2);
                    const int q1 = mino_at<WPL>(E, row * m + q), q2 = mino_at<WPL>(E, rr * m + qq);
                    // entries (row, C2) and (rr, C1) are zeros, (row, C1) and
                    // (rr, C2) nonzeros: one pair by the choice of q1, q2
                    const uint32_t e1 = w_at<WPL>(wbase, st, row, q2), e2 = w_at<WPL>(wbase, st, rr, q1);
                    ok = sparse ? e1 == 1u && e2 == 1u : e1 != 1u && e2 != 1u;
                    x1 = (sparse ? q1 : q2) | ((sparse ? q2 : q1) << 16);
                    pp = q | (qq << 16);
                }
            }
            const unsigned hit = (__ballot_sync(gm, ok) >> base) & ((1u << LPC) - 1u);
            const int src = hit ? base + __ffs((int)hit) - 1 : wl;
            rr = __shfl_sync(gm, rr, src);
            x1 = __shfl_sync(gm, x1, src);
            pp = __shfl_sync(gm, pp, src);
            const uint32_t sw1 = __shfl_sync(gm, d.w, src), sw2 = __shfl_sync(gm, d.x, hit ? src + AT : wl);
            if (pend && hit) {
                kind = 1;
                r2 = rr;
                c1 = x1 & 0xffff;
                c2 = x1 >> 16;
                p1 = pp & 0xffff;
                p2 = pp >> 16;
                s1 = (uint64_t)sw1 < con->thr_swsign;
                s2 = (uint64_t)sw2 < con->thr_swsign;
                pend = false;
            }
            if (!__any_sync(gm, pend)) break;
        }
    }
    if (need && kind < 0) {
        kind = 0;
        r2 = row;
        c1 = c2 = fcol(lds32(cw + 40u), 2, 2, row);
    }
    return make_uint4((uint32_t)row | ((uint32_t)r2 << 16), (uint32_t)c1 | ((uint32_t)c2 << 16),
                      (uint32_t)p1 | ((uint32_t)p2 << 16),
                      (uint32_t)(kind & 3) | (s1 ? 4u : 0u) | (s2 ? 8u : 0u));
}

// A move in three words:
//   rc  R1 | R2<<8 | C1<<16 | C2<<24 (R2 = R1: one row)
//   cf  the coefficients a1, b1 (row R1, columns C1, C2), a2, b2 (row R2)
//   ax  change of G[R1][R2] | p1<<8 | p2<<16 | support change<<24 (bit 0 R1,
//       bit 1 R2), p1, p2 the changed entries of the minority lists; bits
//       26..29 the ninth bits of R1, R2, C1, C2
struct Move {
    uint32_t rc, cf, ax;
};

// A lane's view of its group's candidate: the move, its deltas (score
// change + 4096 x conflict change) and its change of the objective.
struct Cand {
    int R1, R2, C1, C2, p1, p2, kind;
    int a1, b1, a2, b2, pk;
    int acc, prim;
};

template <int WPL>
__device__ __forceinline__ Move pack_move(const Cand& q) {
    Move mv;
    mv.cf = (uint32_t)(q.a1 & 255) | ((uint32_t)(q.b1 & 255) << 8) | ((uint32_t)(q.a2 & 255) << 16) |
            ((uint32_t)q.b2 << 24);
    mv.ax = (uint32_t)(q.pk & 255) | ((uint32_t)q.p1 << 8) | ((uint32_t)q.p2 << 16) |
            (q.kind == 1 ? 3u << 24 : q.kind == 3 ? 1u << 24 : 0u);
    if constexpr (WPL == 16) {
        mv.rc = (uint32_t)(q.R1 & 255) | ((uint32_t)(q.R2 & 255) << 8) | ((uint32_t)(q.C1 & 255) << 16) |
                ((uint32_t)q.C2 << 24);
        mv.ax |= ((uint32_t)(q.R1 >> 8) << 26) | ((uint32_t)(q.R2 >> 8) << 27) | ((uint32_t)(q.C1 >> 8) << 28) |
                 ((uint32_t)(q.C2 >> 8) << 29);
    } else {
        mv.rc = (uint32_t)q.R1 | ((uint32_t)q.R2 << 8) | ((uint32_t)q.C1 << 16) | ((uint32_t)q.C2 << 24);
    }
    return mv;
}

__device__ __forceinline__ Move move_of(const Move& mv, int src, unsigned gm) {
    Move r;
    r.rc = __shfl_sync(gm, mv.rc, src);
    r.cf = __shfl_sync(gm, mv.cf, src);
    r.ax = __shfl_sync(gm, mv.ax, src);
    return r;
}

// v << s, 0 for s >= 32 (also for a "negative" s)
__device__ __forceinline__ uint32_t shl_clamp(uint32_t v, uint32_t s) {
    uint32_t r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(s));
    return r;
}

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

// New halfwords of rows 8j .. 8j+7 of the changed Gram rows of a move above
// order 128: g1, g2 updated in place from the move's coefficients.
__device__ __forceinline__ void wide_rows(uint32_t w1, uint32_t w2, int R1, int R2, int j, int a1, int b1, int a2,
                                          int b2, int pk, uint32_t (&g1)[4], uint32_t (&g2)[4]) {
    const uint2 x8 = *reinterpret_cast<const uint2*>(xw_smem + w1 + 8u * (uint32_t)j);
    const uint2 y8 = *reinterpret_cast<const uint2*>(xw_smem + w2 + 8u * (uint32_t)j);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const uint32_t sel = h & 1 ? 0x4342u : 0x4140u;
        const uint32_t x = __byte_perm(h < 2 ? x8.x : x8.y, 0u, sel), y = __byte_perm(h < 2 ? y8.x : y8.y, 0u, sel);
        // entries R1 and R2 are left out: their W reads as zero (biased 1)
        const uint32_t h1 = 16u * (uint32_t)R1 - 128u * (uint32_t)j - 32u * h,
                       h2 = 16u * (uint32_t)R2 - 128u * (uint32_t)j - 32u * h;
        const uint32_t mm = shl_clamp(0xffffu, h1) | shl_clamp(0xffffu, h2);
        const uint32_t xx = ((x & ~mm) | (0x00010001u & mm)) - 0x00010001u;
        const uint32_t yy = ((y & ~mm) | (0x00010001u & mm)) - 0x00010001u;
        g1[h] += (uint32_t)a1 * xx + (uint32_t)b1 * yy + shl_clamp((uint32_t)pk, h2);
        g2[h] += (uint32_t)a2 * xx + (uint32_t)b2 * yy;
    }
}

// |v| of both biased halfwords
__device__ __forceinline__ uint32_t abs_halves(uint32_t v) {
    const uint32_t t = v ^ 0x80008000u;
    uint32_t m;   // the sign of each half
    asm("prmt.b32 %0, %1, %1, 0xbb99;" : "=r"(m) : "r"(t));
    return (t ^ m) + (m & 0x00010001u);
}

// The sums of eight entries of two changed rows: score + 4096 x conflicts,
// and the change of the squared or parity objective.
template <bool GEN>
__device__ __forceinline__ void wide_sums(int obj_kind, const uint32_t (&g1)[4], const uint32_t (&g2)[4],
                                          const uint32_t (&old1)[4], const uint32_t (&old2)[4], int& acc, int& pr) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const uint32_t v1 = abs_halves(g1[h]), v2 = abs_halves(g2[h]);
        const uint32_t z = (((v1 + 0x7fff7fffu) & 0x80008000u) >> 15) + (((v2 + 0x7fff7fffu) & 0x80008000u) >> 15);
        acc = __dp2a_lo((int)(v1 + v2), 0x0101, acc);   // at most 896 a half
        acc = __dp2a_lo((int)(z << 12), 0x0101, acc);   // 4096 a conflict
        if (GEN) {
            if (obj_kind == 1) {
                auto sq = [](uint32_t a) -> int {
                    const int lo = (int)(a & 0xffffu) - 32768, hi = (int)(a >> 16) - 32768;
                    return lo * lo + hi * hi;
                };
                pr += sq(g1[h]) + sq(g2[h]) - sq(old1[h]) - sq(old2[h]);
            } else if (obj_kind == 2) {
                pr += __popc((g1[h] & 0x00010001u) | ((g2[h] & 0x00010001u) << 1)) -
                      __popc((old1[h] & 0x00010001u) | ((old2[h] & 0x00010001u) << 1));
            }
        }
    }
}

template <bool GEN>
__device__ __forceinline__ void wide_chunk(const Env& E, uint32_t w1, uint32_t w2, int R1, int R2, int j,
                                           const Cand& q, int& acc, int& pr) {
    const uint4 o1 = lds128(wide_at(E.g, E.gst, R1, j)), o2 = lds128(wide_at(E.g, E.gst, R2, j));
    const uint32_t old1[4] = {o1.x, o1.y, o1.z, o1.w}, old2[4] = {o2.x, o2.y, o2.z, o2.w};
    uint32_t g1[4] = {o1.x, o1.y, o1.z, o1.w}, g2[4] = {o2.x, o2.y, o2.z, o2.w};
    wide_rows(w1, w2, R1, R2, j, q.a1, q.b1, q.a2, q.b2, q.pk, g1, g2);
    wide_sums<GEN>(E.obj_kind, g1, g2, old1, old2, acc, pr);
}

// Hybrid form: new halfwords of chunk j of the changed rows, as wide_rows;
// entries R1 and R2 are left out of both columns.  `sym`: the change of
// G[R1][R2] goes into row R2's entry too (a commit writes both).
__device__ __forceinline__ void hybrid_chunk(uint32_t w1, uint32_t w2, int R1, int R2, int j, int a1, int b1, int a2,
                                             int b2, int pk, bool sym, uint32_t (&g1)[4], uint32_t (&g2)[4]) {
    auto bits = [&](int R) -> uint32_t { return (R >> 3) == j ? 0x11u << ((R & 3) + 2 * (R & 4)) : 0u; };
    const uint32_t keep = ~(bits(R1) | bits(R2));
    const uint32_t x = *reinterpret_cast<const uint16_t*>(xw_smem + w1 + 2u * (uint32_t)j) & keep;
    const uint32_t y = *reinterpret_cast<const uint16_t*>(xw_smem + w2 + 2u * (uint32_t)j) & keep;
    const uint2 xa = *reinterpret_cast<const uint2*>(xw_smem + 8u * (x & 255u)),
                xb = *reinterpret_cast<const uint2*>(xw_smem + 8u * (x >> 8));
    const uint2 ya = *reinterpret_cast<const uint2*>(xw_smem + 8u * (y & 255u)),
                yb = *reinterpret_cast<const uint2*>(xw_smem + 8u * (y >> 8));
    const uint32_t X[4] = {xa.x, xa.y, xb.x, xb.y}, Y[4] = {ya.x, ya.y, yb.x, yb.y};
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const uint32_t o = 128u * (uint32_t)j + 32u * h;
        g1[h] += (uint32_t)a1 * X[h] + (uint32_t)b1 * Y[h] + shl_clamp((uint32_t)pk, 16u * (uint32_t)R2 - o);
        g2[h] += (uint32_t)a2 * X[h] + (uint32_t)b2 * Y[h] + (sym ? shl_clamp((uint32_t)pk, 16u * (uint32_t)R1 - o) : 0u);
    }
}

// Entry `e` of the tables of nibble pairs: four entries of W (low nibble
// support, high nibble sign) as the sum of w_i 256^i, or of w_i 65536^i of
// each two.
__device__ __forceinline__ uint32_t nibble_entry_bytes(uint32_t e) {
    uint32_t x = 0;
    for (int i = 3; i >= 0; --i) x = x * 256u + ((e >> i) & 1u) - 2u * ((e >> (4 + i)) & 1u);
    return x;
}

__device__ __forceinline__ uint2 nibble_entry(uint32_t e) {
    auto w = [&](int i) -> int { return (int)((e >> i) & 1u) - 2 * (int)((e >> (4 + i)) & 1u); };
    return make_uint2((uint32_t)w(0) + ((uint32_t)w(1) << 16), (uint32_t)w(2) + ((uint32_t)w(3) << 16));
}

// The same from a G in bytes: new bytes of the 16 entries of chunk j.
__device__ __forceinline__ void hybrid_chunk_bytes(uint32_t w1, uint32_t w2, int R1, int R2, int j, int a1, int b1,
                                                   int a2, int b2, int pk, bool sym, uint32_t (&g1)[4],
                                                   uint32_t (&g2)[4]) {
    auto bits = [&](int R) -> uint32_t { return (R >> 4) == j ? 0x11u << ((R & 3) + 2 * (R & 12)) : 0u; };
    const uint32_t keep = ~(bits(R1) | bits(R2));
    const uint32_t x = lds32(w1 + 4u * (uint32_t)j) & keep, y = lds32(w2 + 4u * (uint32_t)j) & keep;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const uint32_t X = lds32(2048u + 4u * ((x >> (8 * h)) & 255u)), Y = lds32(2048u + 4u * ((y >> (8 * h)) & 255u));
        const uint32_t o = 128u * (uint32_t)j + 32u * h;
        g1[h] += (uint32_t)a1 * X + (uint32_t)b1 * Y + shl_clamp((uint32_t)pk, 8u * (uint32_t)R2 - o);
        g2[h] += (uint32_t)a2 * X + (uint32_t)b2 * Y + (sym ? shl_clamp((uint32_t)pk, 8u * (uint32_t)R1 - o) : 0u);
    }
}

// The lane's 16-byte chunks l, l + 8, ... of a candidate from a G in bytes.
// `over`: a row read holds an entry above kByteMax (the sums are then void).
template <bool GEN>
__device__ __forceinline__ void hybrid_rows_bytes(const Env& E, uint32_t w1, uint32_t w2, int R1, int R2, int l,
                                                  const Cand& q, int& acc, int& pr, bool& over) {
    constexpr int kFlight = 4;   // chunks of both rows in flight (all of them: n <= 512)
    const int nch = (E.n + 15) >> 4;
    const uint32_t bst = hybrid_byte_stride(E.n);
    const uint8_t* p1 = E.gp + (size_t)R1 * bst;
    const uint8_t* p2 = E.gp + (size_t)R2 * bst;
    const bool two = R2 != R1;
    uint4 o1[kFlight], o2[kFlight];
#pragma unroll
    for (int k = 0; k < kFlight; ++k) {
        const int j = l + 8 * k;
        o1[k] = make_uint4(0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u);
        if (j < nch) o1[k] = __ldcg(reinterpret_cast<const uint4*>(p1) + j);
        o2[k] = o1[k];
        if (two && j < nch) o2[k] = __ldcg(reinterpret_cast<const uint4*>(p2) + j);
    }
    uint32_t big = 0, ac = (uint32_t)acc;
#pragma unroll
    for (int k = 0; k < kFlight; ++k) {
        const int j = l + 8 * k;
        if (j < nch) {
            const uint32_t old1[4] = {o1[k].x, o1[k].y, o1[k].z, o1[k].w};
            const uint32_t old2[4] = {o2[k].x, o2[k].y, o2[k].z, o2[k].w};
            uint32_t g1[4] = {o1[k].x, o1[k].y, o1[k].z, o1[k].w}, g2[4] = {o2[k].x, o2[k].y, o2[k].z, o2[k].w};
            hybrid_chunk_bytes(w1, w2, R1, R2, j, q.a1, q.b1, q.a2, q.b2, q.pk, false, g1, g2);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const uint32_t m1 = __vabsdiffu4(old1[h], 0x80808080u), m2 = __vabsdiffu4(old2[h], 0x80808080u);
                big |= (m1 + (uint32_t)(127 - kByteMax) * 0x01010101u) | (m2 + (uint32_t)(127 - kByteMax) * 0x01010101u);
                const uint32_t v1 = __vabsdiffu4(g1[h], 0x80808080u), v2 = __vabsdiffu4(g2[h], 0x80808080u);
                const uint32_t z1 = (v1 + 0x7f7f7f7fu) & 0x80808080u, z2 = (v2 + 0x7f7f7f7fu) & 0x80808080u;
                ac = __dp4a(v1, 0x01010101u, ac);
                ac = __dp4a(v2, 0x01010101u, ac);
                ac = __dp4a(z1, 0x20202020u, ac);   // 128 * 32: 4096 a conflict
                ac = __dp4a(z2, 0x20202020u, ac);
                if (GEN) {
                    if (E.obj_kind == 1) {
                        const int d1 = (int)(g1[h] ^ 0x80808080u), d2 = (int)(g2[h] ^ 0x80808080u);
                        const int e1 = (int)(old1[h] ^ 0x80808080u), e2 = (int)(old2[h] ^ 0x80808080u);
                        pr += __dp4a(d1, d1, 0) + __dp4a(d2, d2, 0) - __dp4a(e1, e1, 0) - __dp4a(e2, e2, 0);
                    } else if (E.obj_kind == 2) {
                        pr += __popc((g1[h] & 0x01010101u) | ((g2[h] & 0x01010101u) << 1)) -
                              __popc((old1[h] & 0x01010101u) | ((old2[h] & 0x01010101u) << 1));
                    }
                }
            }
        }
    }
    acc = (int)ac;
    over = (big & 0x80808080u) != 0u;
}

// G from bytes to halfwords, in place: rows from the last, each read whole
// before its (longer, later) place is written.
__device__ __noinline__ void widen_gram(uint8_t* gp, int n, int lane) {
    const uint32_t bst = hybrid_byte_stride(n), hst = hybrid_gram_stride(n);
#pragma unroll 1
    for (int r = n - 1; r >= 0; --r) {
        uint32_t w[4];   // words lane, lane + 32, ... of the row
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t i = (uint32_t)(lane + 32 * k);
            w[k] = 4u * i < bst ? __ldcg(reinterpret_cast<const uint32_t*>(gp + (size_t)r * bst) + i) : 0x80808080u;
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t i = (uint32_t)(lane + 32 * k);
            if (8u * i < hst) {
                const uint32_t lo = __byte_perm(w[k], 0u, 0x4140u) + 0x7f807f80u, hi = __byte_perm(w[k], 0u, 0x4342u) + 0x7f807f80u;
                *reinterpret_cast<uint2*>(gp + (size_t)r * hst + 8u * i) = make_uint2(lo, hi);
            }
        }
        __syncwarp();
    }
}

// The lane's chunks l, l + 8, ... of a candidate in the hybrid form: the
// Gram rows come from HBM or L2, kFlight chunks of both rows in flight
// before the first is used (all of them up to order 320).
template <bool GEN>
__device__ __forceinline__ void hybrid_rows(const Env& E, uint32_t w1, uint32_t w2, int R1, int R2, int l,
                                            const Cand& q, int& acc, int& pr) {
    constexpr int kFlight = 5;
    const int nch = (E.n + 7) >> 3;
    const uint8_t* p1 = E.gp + (size_t)R1 * E.gst;
    const uint8_t* p2 = E.gp + (size_t)R2 * E.gst;
    const bool two = R2 != R1;
#pragma unroll 1
    for (int j0 = l; j0 < nch; j0 += 8 * kFlight) {
        uint4 o1[kFlight], o2[kFlight];
#pragma unroll
        for (int k = 0; k < kFlight; ++k) {
            const int j = j0 + 8 * k;
            o1[k] = make_uint4(0, 0, 0, 0);
            if (j < nch) o1[k] = __ldcg(reinterpret_cast<const uint4*>(p1) + j);
            o2[k] = o1[k];
            if (two && j < nch) o2[k] = __ldcg(reinterpret_cast<const uint4*>(p2) + j);
        }
#pragma unroll
        for (int k = 0; k < kFlight; ++k) {
            const int j = j0 + 8 * k;
            if (j < nch) {
                const uint32_t old1[4] = {o1[k].x, o1[k].y, o1[k].z, o1[k].w};
                const uint32_t old2[4] = {o2[k].x, o2[k].y, o2[k].z, o2[k].w};
                uint32_t g1[4] = {o1[k].x, o1[k].y, o1[k].z, o1[k].w}, g2[4] = {o2[k].x, o2[k].y, o2[k].z, o2[k].w};
                hybrid_chunk(w1, w2, R1, R2, j, q.a1, q.b1, q.a2, q.b2, q.pk, false, g1, g2);
                wide_sums<GEN>(E.obj_kind, g1, g2, old1, old2, acc, pr);
            }
        }
    }
}

// The candidate of this lane's group: hot-row tournament, proposal and
// evaluation of candidate `c` of iteration it + d_it against the replica's
// current state, from the draw blocks at E.cw.  Groups with act false go
// through the same steps on whatever their blocks hold.
template <int WPL, bool GEN, int GW, bool ONEZ>
__device__ __forceinline__ Cand candidate(const Env& E, uint64_t it, int d_it, int c, bool act, int lane) {
    constexpr int LPC = GW / 4;
    const unsigned gm = group_mask<GW>();
    const int n = E.n, m = ONEZ ? 1 : E.m, sparse = ONEZ ? 0 : E.sparse;
    const uint32_t st = E.st, slot = E.slot, wbase = wbase_of<WPL>(E.slot, E.n), cw = E.cw;
    const Con* con = con_of<WPL>(slot);
    const int l = lane & (LPC - 1);
    Cand q;

    bool edge = false;   // a draw met Lemire's rejection test: take the exact proposal
    auto ix = [&](uint32_t wd, uint32_t cnt) -> int {
        const uint64_t p = (uint64_t)wd * cnt;
        edge = edge || (uint32_t)p < cnt;
        return (int)(p >> 32);
    };
    // C: hot-row tournament, one sample a lane (up to eight samples)
    int hot;
    if (GW == 32 && E.ts <= 8) {
        const uint32_t r = (uint32_t)ix(lds32(cw + 64u + 4u * (uint32_t)l), (uint32_t)n);
        uint32_t key = (lds32(slot + Slot<WPL>::res + 4u * r) << 14) | ((uint32_t)(63 - l) << 8) | (r & 255u);
        if (l >= E.ts) key = 0;
        hot = best_row<WPL, LPC>(key, r, gm);
    } else {
        // (past eight samples each has a Philox block to itself: no
        // tournament when no candidate takes its row.  1028 replicas of
        // W(23,22), 64 samples, a target fraction of 0, 400 iterations: 0.74 ms
        // against 1.56, and 0.92 in a kernel of one row a lane.  Orders above
        // 128 always run it: the test costs every move of theirs 0.6-1%)
        hot = 0;
        if (WPL >= 8 || E.ts <= 8 || __any_sync(gm, act && lds32(cw) < con->coins.x))
            hot = tournament<WPL, GW>(slot, cw, n, E.ts, c, it + (uint64_t)d_it, l, gm);
    }

    // D: the first attempt of the proposal (propose_move,
    // xweigh_cuda.cu:423-447)
    const uint4 b0 = lds128(cw), coins = con->coins;
    const int rdraw = ix(b0.y, (uint32_t)n);
    int R1 = b0.x < coins.x ? hot : rdraw;
    const bool dbl = b0.z < coins.y;
    // (the coin's 32 bits leave out the largest draw of a certain flip: the
    // exact proposal sees to it, and a row swap, which has none, must not
    // begin)
    bool flip = b0.w < coins.z;
    if (!ONEZ || GEN) flip = flip || E.flips;
    flip = flip && !dbl;
    const bool rowswap = GEN && E.move_set == 1 && !flip && !dbl;
    const uint4 b1 = lds128(cw + 16), b2 = lds128(cw + 32), b3 = lds128(cw + 48);
    const int r2d = ix(dbl ? b3.y : b1.y, (uint32_t)(dbl ? n : n - 1));
    int R2 = dbl ? (b3.x < 0x80000000u ? R1 : r2d) : r2d + (r2d >= R1 ? 1 : 0);
    if (flip || rowswap) R2 = R1;
    int C1, C2, p1 = 0, p2 = 0;
    bool bad;
    if constexpr (ONEZ) {
        // the row's only zero is its minority entry
        const int z1 = mino_at<WPL>(E, R1), z2 = mino_at<WPL>(E, R2);
        const int f1 = after_zero(ix(dbl ? b2.w : b1.x, (uint32_t)n), z1, n), f2 = after_zero(ix(b3.z, (uint32_t)n), z2, n);
        const bool sw = !dbl && !flip;
        C1 = sw ? z2 : f1;
        C2 = sw ? z1 : dbl ? f2 : f1;
        bad = flip ? false : (R2 == R1 || sw) && C1 == C2;
    } else {
        auto fcol = [&](uint32_t wd, int row) -> int {
            const int i = ix(wd, (uint32_t)(sparse ? m : n));
            return sparse ? mino_at<WPL>(E, row * m + i) : mask_first<WPL>(slot, row, i, n);
        };
        const int f1 = fcol(dbl ? b2.w : b1.x, R1);
        const int f2 = fcol(b3.z, R2);
        p1 = ix(b1.z, (uint32_t)m);
        p2 = ix(b1.w, (uint32_t)m);
        const int q1 = mino_at<WPL>(E, R1 * m + p1), q2 = mino_at<WPL>(E, R2 * m + p2);
        const uint32_t e1 = w_at<WPL>(wbase, st, R1, q2), e2 = w_at<WPL>(wbase, st, R2, q1);
        const bool illegal = sparse ? e1 != 1u || e2 != 1u : e1 == 1u || e2 == 1u;
        const bool sw = !dbl && !flip;
        C1 = sw ? (sparse ? q1 : q2) : f1;
        C2 = sw ? (sparse ? q2 : q1) : dbl ? f2 : f1;
        bad = sw ? illegal : dbl && R2 == R1 && C1 == C2;
    }
    bool s1 = b2.x < coins.w, s2 = b2.y < coins.w;
    // 2^32 - 1 may lie below a threshold of 2^32
    edge = edge || max(max(max(b0.x, b0.z), max(b0.w, b2.x)), b2.y) == 0xffffffffu;
    int kind = dbl ? 2 : flip ? 0 : 1;
    if (rowswap) {
        kind = 3;
        bad = false;
    }
    if (__any_sync(gm, act && (bad || edge))) {
        // (a tournament's edge shows in one lane of the group)
        const bool need = (__ballot_sync(gm, act && (bad || edge)) >> ((threadIdx.x & 31u) - (uint32_t)l)) & ((1u << LPC) - 1u);
        const bool exact = __any_sync(gm, edge);
        if (exact) hot = tournament<WPL, GW>(slot, cw, n, E.ts, c, it + (uint64_t)d_it, l, gm);
        const uint4 x = propose_exact<WPL, GW, ONEZ>(E, need, exact ? 0 : 1, hot, c, it + (uint64_t)d_it, l);
        if (need) {
            R1 = (int)(x.x & 0xffffu);
            if (kind != 3) {
                R2 = (int)(x.x >> 16);
                C1 = (int)(x.y & 0xffffu);
                C2 = (int)(x.y >> 16);
                p1 = (int)(x.z & 0xffffu);
                p2 = (int)(x.z >> 16);
                kind = (int)(x.w & 3u);
                s1 = (x.w >> 2) & 1u;
                s2 = (x.w >> 3) & 1u;
            }
        }
    }
    if (GEN && kind == 3) {
        // the within-row swap: a nonzero of the row moves to one of its zeros
        const uint32_t dsl = cand_slot(c, 1);
        const int pos = (int)draw_index(sparse ? b1.y : b1.z, (uint32_t)m, dsl, it + (uint64_t)d_it, con->stream, con->k0, con->k1,
                                        sparse ? 1 : 2);
        const int start = (int)draw_index(sparse ? b1.z : b1.y, (uint32_t)n, dsl, it + (uint64_t)d_it, con->stream, con->k0, con->k1,
                                          sparse ? 2 : 1);
        const int z = mino_at<WPL>(E, R1 * m + pos);
        p1 = pos;
        R2 = R1;
        if constexpr (ONEZ) {
            C1 = after_zero(start, z, n);
            C2 = z;
        } else {
            C1 = sparse ? z : mask_first<WPL>(slot, R1, start, n);
            C2 = sparse ? mask_first<WPL, true>(slot, R1, start, n) : z;
        }
        s1 = b1.w < 0x80000000u;
    }

    // E: coefficients, then the new values of the lane's rows
    const uint32_t w1 = wbase + (uint32_t)C1 * st, w2 = wbase + (uint32_t)C2 * st;
    const bool lact = WPL >= 8 || 4 * WPL * l < n;               // the lane holds rows below n
    const uint32_t loff = lact ? (uint32_t)(4 * WPL * l) : 0u;   // their byte offset
    constexpr int NW = WPL >= 8 ? 1 : WPL;
    uint32_t x[NW], y[NW], g1[NW], g2[NW];
    if constexpr (WPL < 8) {
        load_words<WPL>(w1 + loff, x);
        load_words<WPL>(w2 + loff, y);
        load_words<WPL>(E.g + (uint32_t)R1 * st + loff, g1);
        load_words<WPL>(E.g + (uint32_t)R2 * st + loff, g2);
    }
    const uint32_t rs1 = lds32(slot + Slot<WPL>::res + 4u * (uint32_t)R1);
    const uint32_t rs2 = lds32(slot + Slot<WPL>::res + 4u * (uint32_t)R2);
    const int e11 = (int)w_at<WPL>(wbase, st, R1, C1) - 1, e22 = (int)w_at<WPL>(wbase, st, R2, C2) - 1;
    const bool two = R2 != R1, sw = kind == 1, pair = kind == 2 && two;
    const int m11 = sw || (GEN && kind == 3) ? -e11 : -2 * e11, m22 = sw ? -e22 : -2 * e22;
    q.a1 = m11;
    q.b1 = sw ? (s1 ? m11 : -m11) : kind == 2 && !two ? m22 : 0;
    q.a2 = sw ? (s2 ? m22 : -m22) : 0;
    q.b2 = sw || pair ? m22 : 0;
    if (GEN && kind == 3) q.b1 = s1 ? 1 : -1;
    {
        // double flip over two rows (xweigh_cuda.cu:564-583): G[R1][R2]
        const int e21 = (int)w_at<WPL>(wbase, st, R2, C1) - 1, e12 = (int)w_at<WPL>(wbase, st, R1, C2) - 1;
        const int pk = m11 * e21 + m22 * (e12 + (C1 == C2 ? m11 : 0));
        q.pk = pair ? pk : 0;
    }
    int acc = 0, pr = 0;
    const uint32_t s8 = (uint32_t)(32 * WPL * l);   // bit offset of the lane's first row
    if constexpr (WPL == 8) {
        // chunks l, l + 8, ... of eight rows
#pragma unroll 1
        for (int j = l; 8 * j < n; j += 8)
            wide_chunk<GEN>(E, w1, w2, R1, R2, j, q, acc, pr);
    } else if constexpr (WPL == 16) {
        bool halves = con->halves != 0;
        if (!halves) {
            bool over = false;
            if (act) hybrid_rows_bytes<GEN>(E, w1, w2, R1, R2, l, q, acc, pr, over);
            if (__any_sync(FULL, over)) {
                widen_gram(E.gp, n, lane);
                if (lane == 0) con_of<WPL>(slot)->halves = 1;
                __syncwarp();
                halves = true;
                acc = 0;
                pr = 0;
            }
        }
        if (halves && act) hybrid_rows<GEN>(E, w1, w2, R1, R2, l, q, acc, pr);
    } else
#pragma unroll
    for (int j = 0; j < NW; ++j) {
        // columns R1 and R2 of the changed rows are left out (the entry of a
        // double flip over two rows apart): their W reads as zero
        const uint32_t h1 = 8u * (uint32_t)R1 - s8 - 32u * j, h2 = 8u * (uint32_t)R2 - s8 - 32u * j;
        const uint32_t mm = shl_clamp(0xffu, h1) | shl_clamp(0xffu, h2);
        const uint32_t xx = ((x[j] & ~mm) | (0x01010101u & mm)) - 0x01010101u;
        const uint32_t yy = ((y[j] & ~mm) | (0x01010101u & mm)) - 0x01010101u;
        const uint32_t n1 = g1[j] + (uint32_t)q.a1 * xx + (uint32_t)q.b1 * yy + shl_clamp((uint32_t)q.pk, h2);
        const uint32_t n2 = g2[j] + (uint32_t)q.a2 * xx + (uint32_t)q.b2 * yy;
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
    if (!lact) {
        acc = 0;
        pr = 0;
    }
    // less the rows' old sums (their conflicts weigh 4096 here, 2^18 there)
    if (l == 0) {
        if constexpr (WPL == 16) {   // (two rows' sums do not fit 18 bits)
            acc -= (int)rs1 - (int)(rs1 >> kConfShift) * ((1 << kConfShift) - 4096);
            acc -= (int)rs2 - (int)(rs2 >> kConfShift) * ((1 << kConfShift) - 4096);
        } else {
            const uint32_t rs = rs1 + rs2;
            acc -= (int)rs - (int)(rs >> kConfShift) * ((1 << kConfShift) - 4096);
        }
    }
#pragma unroll
    for (int d = 1; d < LPC; d <<= 1) acc += __shfl_xor_sync(gm, acc, d);
    if (GEN && E.obj_kind != 0) {
#pragma unroll
        for (int d = 1; d < LPC; d <<= 1) pr += __shfl_xor_sync(gm, pr, d);
    } else {
        pr = acc - ((acc + 2048) >> 12) * 4096;
    }
    q.R1 = R1;
    q.R2 = R2;
    q.C1 = C1;
    q.C2 = C2;
    q.p1 = p1;
    q.p2 = p2;
    q.kind = kind;
    q.acc = acc;
    q.prim = pr;
    return q;
}

// The least (objective, score, conflicts, index) over the groups with `act`
// (by_index: the least index), as two ordered words, B's low five bits the
// group; all ones when there is none.
__device__ __forceinline__ void best_keys(bool gen_obj, const Cand& q, bool act, int g, bool by_index, unsigned gm,
                                          uint32_t& A, uint32_t& B) {
    const int dc = (q.acc + 2048) >> 12, ds = q.acc - dc * 4096;
    const uint32_t low = ((uint32_t)(ds + 2048) << 16) | ((uint32_t)(dc + 1024) << 5) | (uint32_t)g;
    if (!gen_obj) {
        const uint32_t ka = by_index ? (uint32_t)g : low;
        A = __reduce_min_sync(gm, act ? ka : 0xffffffffu);
        B = A;
    } else {
        const uint32_t ka = by_index ? (uint32_t)g : (uint32_t)(q.prim + (1 << 22));
        A = __reduce_min_sync(gm, act ? ka : 0xffffffffu);
        B = __reduce_min_sync(gm, act && ka == A ? low : 0xffffffffu);
    }
}

// draw_block with the replica's round keys from the slot: five broadcast
// reads in place of the eighteen additions of the key schedule.
__device__ __forceinline__ uint4 philox_keys(uint32_t slot, uint64_t it, uint32_t stream, const uint4* keys) {
    uint4 c = make_uint4(slot, (uint32_t)it, (uint32_t)(it >> 32), stream);
#pragma unroll
    for (int r = 0; r < 5; ++r) {
        const uint4 k = keys[r];
        c = philox_round(c, k.x, k.y);
        c = philox_round(c, k.z, k.w);
    }
    return c;
}

// Fills the draw buffer of a group: block b of candidate c0 + i of
// iteration `it` (multi), or of candidate 0 of iteration it + i (a run of
// one-candidate iterations), i = 0..3, as block i*bpc + b.  MOVE: the
// move-level block of iteration `it` goes into block 24.
template <int GW, bool MOVE = false>
__device__ __forceinline__ void fill_draws(const Env& E, const Con* con, uint64_t it, int c0, bool multi, int lane) {
    uint4* dbuf = reinterpret_cast<uint4*>(xw_smem + E.draws);
#pragma unroll
    for (int h = 0; h < (GW == 16 ? 2 : 1); ++h) {
        const int qb = lane + 16 * h;
        const uint32_t i = E.dq[h] >> 16, b1 = E.dq[h] & 255u;   // b1 = 1 + b
        const uint32_t dslot = MOVE && qb == 24 ? 0u : b1 + (multi ? 128u * ((uint32_t)c0 + i) : 0u);
        const uint4 d = philox_keys(dslot, it + (uint64_t)(multi ? 0u : i), con->stream, con->keys);
        if (qb < (MOVE ? 25 : 24)) dbuf[qb] = d;
    }
}

// The Metropolis test of a change `prim` of the objective with draw `u` at
// the replica's temperature (xweigh_cuda.cu:1040-1060).  Thresholds beyond
// the table are at most one above its last (the products they round lie
// below it), so a draw above that rejects; the rest, and the draw that a
// threshold of 2^32 would need, take the exponential.
template <int WPL>
__device__ __forceinline__ bool accepts_far(uint32_t slot, int prim, uint32_t u) {
    return metropolis_accept(prim, con_of<WPL>(slot)->T, u);
}

template <int WPL>
__device__ __forceinline__ bool accepts(uint32_t slot, int prim, uint32_t u) {
    const int i = min(max(prim, 1), (int)kThrTable);
    const uint32_t t = lds32(slot + Slot<WPL>::thr + 4u * (uint32_t)(i - 1));
    const bool below = u < t || prim <= 0;
    if (prim > 0 && ((prim > (int)kThrTable && u <= t) || u == 0xffffffffu)) return accepts_far<WPL>(slot, prim, u);
    return below;
}

// More than four candidates: the first best of `count` candidates, four a
// pass; the winner's move and deltas in every lane.
struct Winner {
    Move mv;
    int acc, prim, two;   // two: candidates of the iteration that change two rows
};

template <int WPL, bool GEN, int GW, bool ONEZ>
__device__ __forceinline__ Winner choose_many(const Env E, uint64_t it, int count, int lane) {
    constexpr int LPC = GW / 4;
    const unsigned gm = group_mask<GW>();
    const int g = lane / LPC, wl0 = (int)(threadIdx.x & 31u) - lane;
    uint32_t bestA = 0xffffffffu, bestB = 0xffffffffu;
    Winner w{};
#pragma unroll 1
    for (int c0 = 0; c0 < count; c0 += 4) {
        __syncwarp(gm);
        fill_draws<GW>(E, con_of<WPL>(E.slot), it, c0, true, lane);
        __syncwarp(gm);
        const int c = c0 + g;
        const bool act = c < count;
        const Cand q = candidate<WPL, GEN, GW, ONEZ>(E, it, 0, c, act, lane);
        w.two += __popc(__ballot_sync(gm, act && q.R2 != q.R1 && (lane & (LPC - 1)) == 0));
        uint32_t A, B;
        best_keys(GEN && E.obj_kind != 0, q, act, g, false, gm, A, B);
        // a later pass wins only strictly: its candidates come after
        const uint32_t ka = GEN && E.obj_kind != 0 ? A : A >> 5, kb = GEN && E.obj_kind != 0 ? B >> 5 : 0u;
        if (ka < bestA || (ka == bestA && kb < bestB)) {
            bestA = ka;
            bestB = kb;
            const int src = wl0 + (int)(B & 3u) * LPC;
            w.mv = move_of(pack_move<WPL>(q), src, gm);
            w.acc = __shfl_sync(gm, q.acc, src);
            w.prim = __shfl_sync(gm, q.prim, src);
        }
    }
    return w;
}

__device__ __forceinline__ int packed_abs(int v) {
    // |v| and [v != 0] as they count into a packed residual
    return iabs(v) + (v != 0 ? 1 << kConfShift : 0);
}

// Commits a move (commit_*, xweigh_cuda.cu:607-877) whose deltas are `acc`:
// the one or two Gram rows (words, by the first group's lanes) and their
// mirrored columns, the packed residuals, W, the support masks and the
// minority lists.  Lane o owns rows o, o + GW, ... of the columns.
template <int WPL, int GW, bool ONEZ>
__device__ __forceinline__ void commit(const Env& E, const Move& mv, int acc, int lane) {
    constexpr int LPC = GW / 4;
    const unsigned gm = group_mask<GW>();
    const int n = E.n, m = ONEZ ? 1 : E.m, sparse = ONEZ ? 0 : E.sparse;
    const uint32_t st = E.st, slot = E.slot, wbase = E.slot + Slot<WPL>::w;
    const int R1 = (int)(mv.rc & 255u), R2 = (int)((mv.rc >> 8) & 255u);
    const int C1 = (int)((mv.rc >> 16) & 255u), C2 = (int)(mv.rc >> 24);
    const bool two = R2 != R1;
    const uint32_t w1 = wbase + (uint32_t)C1 * st, w2 = wbase + (uint32_t)C2 * st;
    const uint32_t r1 = E.g + (uint32_t)R1 * st, r2 = E.g + (uint32_t)R2 * st;
    // the new rows, as candidate() evaluated them
    const int l = lane & (LPC - 1);
    const bool lact = 4 * WPL * l < n;
    const uint32_t loff = lact ? (uint32_t)(4 * WPL * l) : 0u, s8 = (uint32_t)(32 * WPL * l);
    uint32_t x[WPL], y[WPL], g1[WPL], g2[WPL];
    load_words<WPL>(w1 + loff, x);
    load_words<WPL>(w2 + loff, y);
    load_words<WPL>(r1 + loff, g1);
    load_words<WPL>(r2 + loff, g2);
    {
        const int a1 = (int)(int8_t)(mv.cf & 255u), b1 = (int)(int8_t)((mv.cf >> 8) & 255u);
        const int a2 = (int)(int8_t)((mv.cf >> 16) & 255u), b2 = (int)(int8_t)(mv.cf >> 24);
        const int pk = (int)(int8_t)(mv.ax & 255u);
#pragma unroll
        for (int j = 0; j < WPL; ++j) {
            const uint32_t h1 = 8u * (uint32_t)R1 - s8 - 32u * j, h2 = 8u * (uint32_t)R2 - s8 - 32u * j;
            const uint32_t mm = shl_clamp(0xffu, h1) | shl_clamp(0xffu, h2);
            const uint32_t xx = ((x[j] & ~mm) | (0x01010101u & mm)) - 0x01010101u;
            const uint32_t yy = ((y[j] & ~mm) | (0x01010101u & mm)) - 0x01010101u;
            g1[j] += (uint32_t)a1 * xx + (uint32_t)b1 * yy + shl_clamp((uint32_t)pk, h2);
            g2[j] += (uint32_t)a2 * xx + (uint32_t)b2 * yy;
        }
    }
    uint32_t old[WPL];   // old bytes of rows R1, R2 at the lane's columns
#pragma unroll
    for (int k = 0; k < WPL; ++k) {
        const int o = lane + GW * k;
        old[k] = 0;
        if (o < n) old[k] = (lds8(r1 + (uint32_t)o) << 8) | (lds8(r2 + (uint32_t)o) << 24);
    }
    __syncwarp(gm);
    if (lane < LPC && lact) {
        if constexpr (WPL == 1) {
            *reinterpret_cast<uint32_t*>(xw_smem + r1 + loff) = g1[0];
            if (two) *reinterpret_cast<uint32_t*>(xw_smem + r2 + loff) = g2[0];
        } else if constexpr (WPL == 2) {
            *reinterpret_cast<uint2*>(xw_smem + r1 + loff) = make_uint2(g1[0], g1[1]);
            if (two) *reinterpret_cast<uint2*>(xw_smem + r2 + loff) = make_uint2(g2[0], g2[1]);
        } else {
            *reinterpret_cast<uint4*>(xw_smem + r1 + loff) = make_uint4(g1[0], g1[1], g1[2], g1[3]);
            if (two) *reinterpret_cast<uint4*>(xw_smem + r2 + loff) = make_uint4(g2[0], g2[1], g2[2], g2[3]);
        }
    }
    __syncwarp(gm);
    // columns R1 and R2 (entry (R2, R1) of a double flip over two rows comes
    // from row R1) and the residuals: byte weights +1 new, -1 old
    const int wt1 = 0x0000ff01, wt = two ? (int)0xff01ff01u : wt1;
    int d1[WPL], d[WPL], S1 = 0;
#pragma unroll
    for (int k = 0; k < WPL; ++k) {
        const int o = lane + GW * k;
        d1[k] = d[k] = 0;
        if (o < n) {
            const uint32_t n1 = lds8(r1 + (uint32_t)o), n2 = lds8(r2 + (uint32_t)o);
            const uint32_t col = E.g + (uint32_t)o * st;
            xw_smem[col + (uint32_t)R1] = (uint8_t)n1;
            if (o != R1) xw_smem[col + (uint32_t)R2] = (uint8_t)n2;
            const uint32_t v = __vabsdiffu4(old[k] | n1 | (n2 << 16), 0x80808080u);
            const uint32_t z = ((v + 0x7f7f7f7fu) & 0x80808080u) >> 7;
            d1[k] = __dp4a((int)v, wt1, 0) + (__dp4a((int)z, wt1, 0) << kConfShift);
            d[k] = __dp4a((int)v, wt, 0) + (__dp4a((int)z, wt, 0) << kConfShift);
            S1 += d1[k];
        }
    }
    S1 = __reduce_add_sync(gm, S1);
    const int dc = (acc + 2048) >> 12;
    const int S = acc - dc * 4096 + dc * (1 << kConfShift);   // both rows, the pair entry once
#pragma unroll
    for (int k = 0; k < WPL; ++k) {
        const int o = lane + GW * k;
        if (o < n) {
            int* r = reinterpret_cast<int*>(xw_smem + slot + Slot<WPL>::res) + o;
            *r += o == R1 ? S1 : o == R2 ? S - S1 + d1[k] : d[k];
        }
    }
    // one changed entry of W per lane 0..3
    if (lane < 4) {
        const int cfc = (int)(int8_t)((mv.cf >> (8 * lane)) & 255u);
        if (cfc != 0) {
            const uint32_t a = ((lane & 1) ? w2 : w1) + (uint32_t)((lane & 2) ? R2 : R1);
            xw_smem[a] = (uint8_t)(lds8(a) + (uint32_t)cfc);
        }
        // support mask and minority entry of rows R1 (lane 0) and R2 (lane 1)
        if (lane < 2 && ((mv.ax >> (24 + lane)) & 1u)) {
            const int R = lane ? R2 : R1;
            if constexpr (ONEZ) {
            } else if constexpr (WPL == 1) {
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

// The same above order 128: lane c rewrites chunk c of the two rows, then
// lane o takes rows o, o + 32, ... of the columns.
template <bool ONEZ>
__device__ __forceinline__ void commit_wide(const Env& E, const Move& mv, int acc, int lane) {
    const int n = E.n, m = ONEZ ? 1 : E.m, sparse = ONEZ ? 0 : E.sparse;
    const uint32_t st = E.st, slot = E.slot, wbase = E.slot + Slot<8>::w, g = E.g, gst = E.gst;
    const int R1 = (int)(mv.rc & 255u), R2 = (int)((mv.rc >> 8) & 255u);
    const int C1 = (int)((mv.rc >> 16) & 255u), C2 = (int)(mv.rc >> 24);
    const bool two = R2 != R1;
    const uint32_t w1 = wbase + (uint32_t)C1 * st, w2 = wbase + (uint32_t)C2 * st;
    auto half = [&](int row, int col) -> uint16_t* {
        return reinterpret_cast<uint16_t*>(xw_smem + wide_at(g, gst, row, col >> 3)) + (col & 7);
    };
    uint32_t old1[8], old2[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int o = lane + 32 * k;
        old1[k] = old2[k] = 0;
        if (o < n) {
            old1[k] = *half(R1, o);
            old2[k] = *half(R2, o);
        }
    }
    const bool mine = 8 * lane < n;
    uint32_t g1[4], g2[4];
    if (mine) {
        const uint4 o1 = lds128(wide_at(g, gst, R1, lane)), o2 = lds128(wide_at(g, gst, R2, lane));
        g1[0] = o1.x; g1[1] = o1.y; g1[2] = o1.z; g1[3] = o1.w;
        g2[0] = o2.x; g2[1] = o2.y; g2[2] = o2.z; g2[3] = o2.w;
        wide_rows(w1, w2, R1, R2, lane, (int)(int8_t)(mv.cf & 255u), (int)(int8_t)((mv.cf >> 8) & 255u),
                  (int)(int8_t)((mv.cf >> 16) & 255u), (int)(int8_t)(mv.cf >> 24), (int)(int8_t)(mv.ax & 255u), g1, g2);
    }
    __syncwarp();
    if (mine) {
        *reinterpret_cast<uint4*>(xw_smem + wide_at(g, gst, R1, lane)) = make_uint4(g1[0], g1[1], g1[2], g1[3]);
        if (two) *reinterpret_cast<uint4*>(xw_smem + wide_at(g, gst, R2, lane)) = make_uint4(g2[0], g2[1], g2[2], g2[3]);
    }
    __syncwarp();
    int d1[8], d[8], S1 = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int o = lane + 32 * k;
        d1[k] = d[k] = 0;
        if (o < n) {
            const uint32_t n1 = *half(R1, o), n2 = *half(R2, o);
            *half(o, R1) = (uint16_t)n1;
            if (o != R1) *half(o, R2) = (uint16_t)n2;
            d1[k] = packed_abs((int)n1 - 32768) - packed_abs((int)old1[k] - 32768);
            d[k] = d1[k] + (two ? packed_abs((int)n2 - 32768) - packed_abs((int)old2[k] - 32768) : 0);
            S1 += d1[k];
        }
    }
    S1 = __reduce_add_sync(FULL, S1);
    const int dc = (acc + 2048) >> 12;
    const int S = acc - dc * 4096 + dc * (1 << kConfShift);   // both rows, the pair entry once
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int o = lane + 32 * k;
        if (o < n) {
            int* r = reinterpret_cast<int*>(xw_smem + slot + Slot<8>::res) + o;
            *r += o == R1 ? S1 : o == R2 ? S - S1 + d1[k] : d[k];
        }
    }
    if (lane < 4) {
        const int cfc = (int)(int8_t)((mv.cf >> (8 * lane)) & 255u);
        if (cfc != 0) {
            const uint32_t a = ((lane & 1) ? w2 : w1) + (uint32_t)((lane & 2) ? R2 : R1);
            xw_smem[a] = (uint8_t)(lds8(a) + (uint32_t)cfc);
        }
        if (lane < 2 && ((mv.ax >> (24 + lane)) & 1u)) {
            const int lost = lane ? C2 : C1, got = lane ? C1 : C2;
            const int p = (int)((mv.ax >> (8 + 8 * lane)) & 255u);
            xw_smem[E.mino + (uint32_t)((lane ? R2 : R1) * m + p)] = (uint8_t)(sparse ? got : lost);
        }
    }
}

// Adds `d` to entry (r, c) of a nibble-pair W.
__device__ __forceinline__ void nibble_add(uint32_t wbase, uint32_t st, int r, int c, int d) {
    const uint32_t a = wbase + (uint32_t)c * st + ((uint32_t)r >> 2), b = lds8(a);
    const int i = r & 3, w = (int)((b >> i) & 1u) - 2 * (int)((b >> (4 + i)) & 1u) + d;
    const uint32_t v = (w != 0 ? 1u : 0u) | (w < 0 ? 16u : 0u);
    xw_smem[a] = (uint8_t)((b & ~(0x11u << i)) | (v << i));
}

// Commit in the hybrid form: lane c rewrites chunks c, c + 32 of the two
// rows and the entries of columns R1 and R2 in the rows of those chunks.
__device__ __forceinline__ void commit_hybrid(const Env& E, const Move& mv, int acc, int lane) {
    const int n = E.n, m = E.m, nch = (n + 7) >> 3;
    const uint32_t st = E.st, slot = E.slot, wbase = wbase_of<16>(slot, n);
    const int R1 = (int)((mv.rc & 255u) | ((mv.ax >> 18) & 256u)), R2 = (int)(((mv.rc >> 8) & 255u) | ((mv.ax >> 19) & 256u));
    const int C1 = (int)(((mv.rc >> 16) & 255u) | ((mv.ax >> 20) & 256u)), C2 = (int)((mv.rc >> 24) | ((mv.ax >> 21) & 256u));
    const bool two = R2 != R1;
    const int a1 = (int)(int8_t)(mv.cf & 255u), b1 = (int)(int8_t)((mv.cf >> 8) & 255u);
    const int a2 = (int)(int8_t)((mv.cf >> 16) & 255u), b2 = (int)(int8_t)(mv.cf >> 24);
    const int pk = (int)(int8_t)(mv.ax & 255u);
    int S1 = 0, dpair = 0;
    const bool halves = con_of<16>(slot)->halves != 0;
    if (!halves) {
        // bytes: words lane, lane + 32, ... of both rows, one ahead (a loop
        // of four rows against one pass over sixteen a lane, which left 14
        // lanes of W(276,275) idle and fetched four times the code: 2368
        // replicas 15.3 -> 14.2 ms, 148 replicas 5.1 -> 4.8, 2368 of
        // W(400,200) 41.6 -> 36.9; the same loop for the evaluation's reads,
        // which then wait for each other: 14.7, 5.4 and 40.7)
        const uint32_t bst = hybrid_byte_stride(n);
        uint32_t* q1 = reinterpret_cast<uint32_t*>(E.gp + (size_t)R1 * bst);
        uint32_t* q2 = reinterpret_cast<uint32_t*>(E.gp + (size_t)R2 * bst);
        const uint32_t w1 = wbase + (uint32_t)C1 * st, w2 = wbase + (uint32_t)C2 * st;
        const int nwd = (n + 3) >> 2, wt1 = 0x0000ff01, wt = two ? (int)0xff01ff01u : wt1;
        uint32_t next1 = 0, next2 = 0;
        if (lane < nwd) {
            next1 = __ldcg(q1 + lane);
            next2 = __ldcg(q2 + lane);
        }
#pragma unroll 1
        for (int j = lane; j < nwd; j += 32) {
            const uint32_t old1 = next1, old2 = next2;
            if (j + 32 < nwd) {
                next1 = __ldcg(q1 + j + 32);
                next2 = __ldcg(q2 + j + 32);
            }
            const uint32_t keep = ~((R1 >> 2) == j ? 0x11u << (R1 & 3) : 0u) & ~((R2 >> 2) == j ? 0x11u << (R2 & 3) : 0u);
            const uint32_t X = lds32(2048u + 4u * (lds8(w1 + (uint32_t)j) & keep)),
                           Y = lds32(2048u + 4u * (lds8(w2 + (uint32_t)j) & keep));
            const uint32_t o32 = 32u * (uint32_t)j;
            const uint32_t g1 = old1 + (uint32_t)a1 * X + (uint32_t)b1 * Y + shl_clamp((uint32_t)pk, 8u * (uint32_t)R2 - o32);
            const uint32_t g2 = old2 + (uint32_t)a2 * X + (uint32_t)b2 * Y + shl_clamp((uint32_t)pk, 8u * (uint32_t)R1 - o32);
            q1[j] = g1;
            if (two) q2[j] = g2;
            int* res = reinterpret_cast<int*>(xw_smem + slot + Slot<16>::res) + 4 * j;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int o = 4 * j + i, sh = 8 * i;
                if (o < n) {
                    const uint32_t n1 = (g1 >> sh) & 255u, n2 = (g2 >> sh) & 255u;
                    const uint32_t v = __vabsdiffu4(n1 | (((old1 >> sh) & 255u) << 8) | (n2 << 16) | (((old2 >> sh) & 255u) << 24),
                                                    0x80808080u);
                    const uint32_t z = ((v + 0x7f7f7f7fu) & 0x80808080u) >> 7;
                    const int d1 = __dp4a((int)v, wt1, 0) + (__dp4a((int)z, wt1, 0) << kConfShift);
                    S1 += d1;
                    if (o == R2) dpair = d1;
                    if (o != R1 && o != R2) {
                        uint8_t* row = E.gp + (size_t)o * bst;
                        row[R1] = (uint8_t)n1;
                        if (two) row[R2] = (uint8_t)n2;
                        res[i] += __dp4a((int)v, wt, 0) + (__dp4a((int)z, wt, 0) << kConfShift);
                    }
                }
            }
        }
    }
#pragma unroll 1
    for (int j = halves ? lane : nch; j < nch; j += 32) {
        uint4* q1 = reinterpret_cast<uint4*>(E.gp + (size_t)R1 * E.gst) + j;
        uint4* q2 = reinterpret_cast<uint4*>(E.gp + (size_t)R2 * E.gst) + j;
        const uint4 o1 = __ldcg(q1), o2 = two ? __ldcg(q2) : o1;
        const uint32_t old1[4] = {o1.x, o1.y, o1.z, o1.w}, old2[4] = {o2.x, o2.y, o2.z, o2.w};
        uint32_t g1[4] = {o1.x, o1.y, o1.z, o1.w}, g2[4] = {o2.x, o2.y, o2.z, o2.w};
        hybrid_chunk(wbase + (uint32_t)C1 * st, wbase + (uint32_t)C2 * st, R1, R2, j, a1, b1, a2, b2, pk, true, g1, g2);
        *q1 = make_uint4(g1[0], g1[1], g1[2], g1[3]);
        if (two) *q2 = make_uint4(g2[0], g2[1], g2[2], g2[3]);
        int* res = reinterpret_cast<int*>(xw_smem + slot + Slot<16>::res) + 8 * j;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int o = 8 * j + i, sh = 16 * (i & 1);
            const uint32_t n1 = (g1[i >> 1] >> sh) & 0xffffu, n2 = (g2[i >> 1] >> sh) & 0xffffu;
            const int d1 = packed_abs((int)n1 - 32768) - packed_abs((int)((old1[i >> 1] >> sh) & 0xffffu) - 32768);
            const int d2 = packed_abs((int)n2 - 32768) - packed_abs((int)((old2[i >> 1] >> sh) & 0xffffu) - 32768);
            if (o < n) {
                S1 += d1;
                if (o == R2) dpair = d1;
                // rows R1 and R2 themselves are written by chunks only: a
                // lane may still have to read its chunk of them
                if (o != R1 && o != R2) {
                    uint16_t* row = reinterpret_cast<uint16_t*>(E.gp + (size_t)o * E.gst);
                    row[R1] = (uint16_t)n1;
                    if (two) row[R2] = (uint16_t)n2;
                    res[i] += two ? d1 + d2 : d1;
                }
            }
        }
    }
    S1 = __reduce_add_sync(FULL, S1);
    const int dc = (acc + 2048) >> 12;
    const int S = acc - dc * 4096 + dc * (1 << kConfShift);   // both rows, the pair entry once
    int* res = reinterpret_cast<int*>(xw_smem + slot + Slot<16>::res);
    if ((halves ? (R2 >> 3) & 31 : (R2 >> 2) & 31) == lane && two) res[R2] += S - S1 + dpair;
    if (lane == 0) res[R1] += S1;
    // (every lane has read W's columns; two entries may share a byte)
    __syncwarp();
    if (lane == 0) {
        if (a1) nibble_add(wbase, st, R1, C1, a1);
        if (a2) nibble_add(wbase, st, R2, C1, a2);
    }
    if (lane == (C1 == C2 ? 0 : 1)) {
        if (b1) nibble_add(wbase, st, R1, C2, b1);
        if (b2) nibble_add(wbase, st, R2, C2, b2);
    }
    if (lane < 2 && ((mv.ax >> (24 + lane)) & 1u)) {
        const int lost = lane ? C2 : C1, got = lane ? C1 : C2;
        const int p = (int)((mv.ax >> (8 + 8 * lane)) & 255u);
        E.mp[(lane ? R2 : R1) * m + p] = (uint16_t)(E.sparse ? got : lost);
    }
}

// tab[d-1] = ceil(exp(-d/T) * 2^32), computed with the same division and
// exponential as metropolis_accept, so that for a 32-bit draw u
//   u * 2^-32 < exp(-d/T)  <=>  u < tab[d-1]
// exactly (both sides scaled by 2^32 without rounding; u is an integer).
// 2^32 itself (T above 4e9) is kept as 2^32 - 1 in a 32-bit table.
// Rebuilt whenever the replica's temperature changes.
template <int GW = 32, typename TAB>
__device__ __forceinline__ void build_thresholds(TAB* tab, double T, int lane) {
    const double t = T > 1.0e-12 ? T : 1.0e-12;
    for (uint32_t d = lane + 1; d <= kThrTable; d += GW) {
        const double e = acceptance_exp(__ddiv_rn(-(double)d, t));
        const uint64_t v = (uint64_t)ceil(__dmul_rn(e, 0x1p32));
        tab[d - 1] = sizeof(TAB) == 4 && v > 0xffffffffull ? (TAB)0xffffffffu : (TAB)v;
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

// The replica's W as int8, column-major, into its record: a word (four rows
// of a column) a lane.
template <int WPL, int GW>
__device__ __noinline__ void save_w(int8_t* dst, uint32_t wbase, uint32_t st, int n, int lane) {
    const int wpc = (n + 3) >> 2;
    const bool whole = (n & 3) == 0;   // every word of the record is aligned and full
    if constexpr (WPL == 16) {
        // four entries of column k from nibble pair j: bit i of a nibble to byte i
        auto entries = [&](int k, int j) -> uint32_t {
            const uint32_t x = lds8(wbase + (uint32_t)k * st + (uint32_t)j);
            return (((x & 15u) * 0x00204081u) & 0x01010101u) + (((x >> 4) * 0x00204081u) & 0x01010101u) * 0xfeu;
        };
        // the pairs that are whole, a lane each, by the widest store that n aligns
        auto columns = [&](auto store) {
#pragma unroll 1
            for (int j = lane; j < (n >> 2); j += 32) {
                int8_t* d = dst + 4 * j;
#pragma unroll 4
                for (int k = 0; k < n; ++k, d += n) store(d, entries(k, j));
            }
        };
        if (whole) {
            columns([](int8_t* d, uint32_t v) { *reinterpret_cast<uint32_t*>(d) = v; });
            return;
        }
        if ((n & 1) == 0) {
            columns([](int8_t* d, uint32_t v) {
                reinterpret_cast<uint16_t*>(d)[0] = (uint16_t)v;
                reinterpret_cast<uint16_t*>(d)[1] = (uint16_t)(v >> 16);
            });
        } else {
            columns([](int8_t* d, uint32_t v) {
#pragma unroll
                for (int e = 0; e < 4; ++e) d[e] = (int8_t)(v >> (8 * e));
            });
        }
        // the last rows, a column a lane
#pragma unroll 1
        for (int k = lane; k < n; k += 32) {
            const uint32_t v = entries(k, n >> 2);
            for (int e = 0; e < (n & 3); ++e) dst[(uint32_t)(k * n + (n & ~3) + e)] = (int8_t)(v >> (8 * e));
        }
        return;
    }
    int c = 0, q = lane;
#pragma unroll 1
    for (;;) {
        while (q >= wpc) {
            q -= wpc;
            ++c;
        }
        if (c >= n) break;
        const uint32_t b = ((lds32(wbase + (uint32_t)c * st + 4u * (uint32_t)q) | 0x80808080u) - 0x01010101u) ^ 0x80808080u;
        int8_t* d = dst + (uint32_t)(c * n + 4 * q);
        if (whole) {
            *reinterpret_cast<uint32_t*>(d) = b;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (4 * q + e < n) d[e] = (int8_t)(b >> (8 * e));
        }
        q += GW;
    }
}

// The best W into the record: the journal's `jn` moves taken out of W,
// written, and put back.
template <int WPL, int GW>
__device__ __forceinline__ void save_best(uint8_t* rec, const XwJob* J, const Env& E, int jn, int lane) {
    const unsigned gm = group_mask<GW>();
    const uint32_t wbase = wbase_of<WPL>(E.slot, E.n);
    auto add = [&](int sign) {
        // (out newest first, so that every entry stays ternary on the way)
        for (int k = 0; k < jn; ++k) {
            const int i = sign < 0 ? jn - 1 - k : k;
            const uint2 mv = *reinterpret_cast<const uint2*>(xw_smem + E.slot + Slot<WPL>::jrn + 8u * (uint32_t)i);
            // entry e: row R1 or R2 (bit 1), column C1 or C2 (bit 0)
            auto entry = [&](int e, int& r, int& c) -> int {
                r = (int)(((mv.x >> ((e & 2) ? 8 : 0)) & 255u) | (((mv.y >> ((e & 2) ? 17 : 16)) & 1u) << 8));
                c = (int)(((mv.x >> ((e & 1) ? 24 : 16)) & 255u) | (((mv.y >> ((e & 1) ? 19 : 18)) & 1u) << 8));
                return sign * ((int)(mv.y << (28 - 4 * e)) >> 28);
            };
            int r, c;
            if constexpr (WPL == 16) {
                if (lane == 0) {   // (two entries may share a byte)
                    for (int e = 0; e < 4; ++e) {
                        const int d = entry(e, r, c);
                        if (d) nibble_add(wbase, E.st, r, c, d);
                    }
                }
            } else {
                const int d = entry(lane & 3, r, c);
                if (lane < 4 && d != 0) {
                    const uint32_t a = wbase + (uint32_t)c * E.st + (uint32_t)r;
                    xw_smem[a] = (uint8_t)((int)lds8(a) + d);
                }
            }
            __syncwarp(gm);
        }
    };
    add(-1);
    save_w<WPL, GW>(reinterpret_cast<int8_t*>(rec + J->off_best), wbase, E.st, E.n, lane);
    __syncwarp(gm);
    add(1);
}

// The lane's context, from the job and the slot.
template <int WPL, bool GEN, int GW, bool ONEZ>
__device__ __forceinline__ void make_env(Env& E, const XwJob* J, uint32_t slot, uint32_t draws, int lane, int obj_kind) {
    constexpr int LPC = GW / 4;
    const int n = J->n;
    E.slot = slot;
    E.draws = draws;
    E.n = n;
    E.m = ONEZ ? 1 : J->m;
    E.sparse = ONEZ ? 0 : J->sparse;
    E.flips = (!ONEZ && J->w == n ? 1 : 0) | (GEN ? (int)(J->thr_sign >> 32) : 0);
    E.st = packed_stride(n, WPL);
    E.gst = WPL == 16 ? hybrid_gram_stride(n) : WPL == 8 ? wide_stride(n) : E.st;
    const uint32_t mat = xw_pad16((uint32_t)n * E.st);
    E.g = wbase_of<WPL>(slot, n) + mat;
    E.mino = WPL == 16 ? E.g : E.g + (WPL == 8 ? (uint32_t)n * E.gst : mat);
    E.gp = nullptr;
    E.mp = nullptr;
    E.ts = J->target_samples;
    E.bpc = 4 + (E.ts <= 4 ? 1 : 2);   // cached blocks per candidate
    E.cw = draws + (uint32_t)((lane / LPC) * E.bpc) * 16u;
    E.move_set = J->move_set;
    E.obj_kind = obj_kind;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int i = (lane + 16 * h) / E.bpc;
        E.dq[h] = ((uint32_t)i << 16) | (uint32_t)(1 + lane + 16 * h - i * E.bpc);
    }
}

// The slot's structures from the record's W: biased bytes, support masks,
// minority lists (copied from the record once it holds them), the Gram
// matrix by popcounts of support and sign masks, the packed residuals.
// False when an entry is not ternary or a row's weight is not w.
template <int WPL, int GW>
__device__ __forceinline__ bool build_packed(const Env& E, const XwJob* J, const uint8_t* rec, uint32_t status0, int w,
                                             int lane, int& score0, int& conf0, int& par0, long long& sq0) {
    constexpr int OPL = WPL;   // rows o, o + GW, ... of a lane: GW * OPL >= n
    const unsigned gm = group_mask<GW>();
    const int n = E.n, m = E.m, sparse = E.sparse;
    const uint32_t slot = E.slot, st = E.st, wbase = slot + Slot<WPL>::w;

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
#pragma unroll 4
        for (int c = 32 * q; c < min(n, 32 * q + 32); ++c) {
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
    if (__any_sync(gm, bad)) return false;
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
    score0 = __reduce_add_sync(gm, p_score) / 2;
    conf0 = __reduce_add_sync(gm, p_conf) / 2;
#pragma unroll
    for (int off = GW / 2; off > 0; off >>= 1) p_sq += __shfl_xor_sync(gm, p_sq, off, GW);
    sq0 = p_sq / 2;
    par0 = __reduce_add_sync(gm, p_par) / 2;
    __syncwarp(gm);
    return true;
}

// The same above order 128.  The masks of all rows (support and sign, 64
// bytes a row) sit in the place of the last rows of G while the rows before
// them are computed; those last rows (at most 32) are the transpose of what
// is known by then and a block among themselves.
__device__ __forceinline__ bool build_wide(const Env& E, const XwJob* J, const uint8_t* rec, uint32_t status0, int w,
                                           int lane, int& score0, int& conf0, int& par0, long long& sq0) {
    const int n = E.n, m = E.m, sparse = E.sparse;
    const uint32_t slot = E.slot, st = E.st, wbase = slot + Slot<8>::w, g = E.g, gst = E.gst;
    const int tail = (int)((64u * (uint32_t)n + gst - 1u) / gst), n0 = n - tail;
    const uint32_t masks = g + (uint32_t)n0 * gst;   // row o: words 16 o + q support, + 8 sign
    const int8_t* gw = reinterpret_cast<const int8_t*>(rec + J->off_w);
    int bad = 0;
#pragma unroll 1
    for (int o = lane; o < (int)st; o += 32) {
#pragma unroll 1
        for (int q = 0; 32 * q < n; ++q) {
            uint32_t sup = 0, neg = 0;
            const int c1 = min(n, 32 * q + 32);
#pragma unroll 8
            for (int c = 32 * q; c < c1; ++c) {
                const int v = o < n ? gw[(uint32_t)(c * n + o)] : 0;
                if (v < -1 || v > 1) bad = 1;
                if (v) sup |= 1u << (c & 31);
                if (v < 0) neg |= 1u << (c & 31);
                xw_smem[wbase + (uint32_t)c * st + (uint32_t)o] = (uint8_t)(v + 1);
            }
            if (o < n) {
                reinterpret_cast<uint32_t*>(xw_smem + masks)[16 * o + q] = sup;
                reinterpret_cast<uint32_t*>(xw_smem + masks)[16 * o + 8 + q] = neg;
            }
        }
    }
    if (m == 0 && lane == 0) xw_smem[E.mino] = 0;   // an empty list still reads as column 0
    const int nq = (n + 31) >> 5;
#pragma unroll 1
    for (int o = lane; o < n; o += 32) {
        int weight = 0, pos = 0;
#pragma unroll 1
        for (int q = 0; q < nq; ++q) {
            const uint32_t sup = lds32(masks + 64u * (uint32_t)o + 4u * (uint32_t)q);
            weight += __popc(sup);
            if (m > 0 && !(status0 & XW_STATUS_INIT)) {
                const int left = n - 32 * q;
                uint32_t x = (sparse ? sup : ~sup) & (left >= 32 ? 0xffffffffu : (1u << left) - 1u);
                while (x && pos < m) {
                    xw_smem[E.mino + (uint32_t)(o * m + pos)] = (uint8_t)(32 * q + __ffs((int)x) - 1);
                    x &= x - 1;
                    ++pos;
                }
            }
        }
        if (weight != w) bad = 1;
    }
    if (m > 0 && (status0 & XW_STATUS_INIT)) {
        const uint8_t* gm8 = rec + J->off_mino;
        for (uint32_t i = lane; i < (uint32_t)(n * m); i += 32) xw_smem[E.mino + i] = gm8[i];
    }
    if (__any_sync(FULL, bad)) return false;
    __syncwarp();
    auto half = [&](int row, int col) -> uint16_t* {
        return reinterpret_cast<uint16_t*>(xw_smem + wide_at(g, gst, row, col >> 3)) + (col & 7);
    };
    // the lane's row of the tail, before it is overwritten
    uint32_t ts[8], tn[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        ts[q] = tn[q] = 0;
        if (lane < tail && q < nq) {
            ts[q] = lds32(masks + 64u * (uint32_t)(n0 + lane) + 4u * (uint32_t)q);
            tn[q] = lds32(masks + 64u * (uint32_t)(n0 + lane) + 32u + 4u * (uint32_t)q);
        }
    }
#pragma unroll 1
    for (int o = lane; o < (int)st; o += 32) {
        uint32_t sup[8], neg[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            sup[q] = neg[q] = 0;
            if (o < n && q < nq) {
                sup[q] = lds32(masks + 64u * (uint32_t)o + 4u * (uint32_t)q);
                neg[q] = lds32(masks + 64u * (uint32_t)o + 32u + 4u * (uint32_t)q);
            }
        }
#pragma unroll 2
        for (int r = 0; r < n0; ++r) {
            int dot = 0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4 rs = lds128(masks + 64u * (uint32_t)r + 16u * h), rn = lds128(masks + 64u * (uint32_t)r + 32u + 16u * h);
                if (4 * h < nq) {
                    const uint32_t b0 = sup[4 * h] & rs.x, b1 = sup[4 * h + 1] & rs.y, b2 = sup[4 * h + 2] & rs.z,
                                   b3 = sup[4 * h + 3] & rs.w;
                    dot += __popc(b0) + __popc(b1) + __popc(b2) + __popc(b3) -
                           2 * (__popc(b0 & (neg[4 * h] ^ rn.x)) + __popc(b1 & (neg[4 * h + 1] ^ rn.y)) +
                                __popc(b2 & (neg[4 * h + 2] ^ rn.z)) + __popc(b3 & (neg[4 * h + 3] ^ rn.w)));
                }
            }
            *half(r, o) = (uint16_t)(32768 + (o == r || o >= n ? 0 : dot));
        }
    }
    __syncwarp();
    // the last rows: columns below n0 by symmetry, then the block of the tail
#pragma unroll 1
    for (int r = n0; r < n; ++r)
        for (int o = lane; o < n0; o += 32) *half(r, o) = *half(o, r);
#pragma unroll 1
    for (int t = 0; t < tail; ++t) {
        int dot = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const uint32_t both = ts[q] & __shfl_sync(FULL, ts[q], t);
            dot += __popc(both) - 2 * __popc(both & (tn[q] ^ __shfl_sync(FULL, tn[q], t)));
        }
        const int o = n0 + lane;
        if (lane < tail) *half(n0 + t, o) = (uint16_t)(32768 + (lane == t ? 0 : dot));
        // the row's pad
        for (int c = n + lane; c < (int)st; c += 32) *half(n0 + t, c) = 32768;
    }
    __syncwarp();
    int p_score = 0, p_conf = 0, p_par = 0;
    long long p_sq = 0;
#pragma unroll 1
    for (int o = lane; o < n; o += 32) {
        int r_sum = 0;
#pragma unroll 4
        for (int r = 0; r < n; ++r) {
            const int v = (int)*half(r, o) - 32768;
            r_sum += packed_abs(v);
            p_sq += (long long)(v * v);
            p_par += v & 1;
        }
        reinterpret_cast<int*>(xw_smem + slot + Slot<8>::res)[o] = r_sum;
        p_score += r_sum & ((1 << kConfShift) - 1);
        p_conf += r_sum >> kConfShift;
    }
    score0 = __reduce_add_sync(FULL, p_score) / 2;
    conf0 = __reduce_add_sync(FULL, p_conf) / 2;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) p_sq += __shfl_xor_sync(FULL, p_sq, off);
    sq0 = p_sq / 2;
    par0 = __reduce_add_sync(FULL, p_par) / 2;
    __syncwarp();
    return true;
}

__device__ __forceinline__ void mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// G of the hybrid form, and the packed residuals, from the rows of W as
// signed nibbles: mma.m16n8k32 on bytes, 16 rows against 8 at a time.  A
// nibble in the upper half of a byte is 16 w, so that the products carry a
// factor of 256 and no sign has to be extended; lane t of a quad holds
// columns 64 Q + 16 t .. + 15 of its row in both operands, an order of the
// contraction index that leaves the sums alone.  (By popcounts of row masks
// the same took 18 POPC an entry: 3.9 of 4.9 ms that 2368 replicas of
// W(276,275) took to load, 10 warps on an SM.)  Byte form: true when an
// entry exceeds kByteMax.
__device__ __forceinline__ bool hybrid_gram(bool halves, uint8_t* gp, const uint8_t* rows, int* res, int n, int lane,
                                            int& p_score, int& p_conf, int& p_par, long long& p_sq) {
    constexpr int kMaxK = kHybridMaxOrder / 64;
    const int g = lane >> 2, t = lane & 3, nk = (n + 63) >> 6;
    const uint32_t rst = hybrid_row_stride(n), gst = halves ? hybrid_gram_stride(n) : hybrid_byte_stride(n);
    const int nc = halves ? (n + 7) >> 3 : (int)(gst >> 3);
    bool over = false;
    auto load = [&](int row, uint2 (&x)[kMaxK]) {
        const uint2* p = reinterpret_cast<const uint2*>(rows + (uint32_t)row * rst) + t;
#pragma unroll
        for (int Q = 0; Q < kMaxK; ++Q) {
            x[Q] = make_uint2(0u, 0u);
            if (Q < nk && row < n) x[Q] = __ldcg(p + 4 * Q);
        }
    };
    auto lo = [](uint32_t x) -> uint32_t { return (x << 4) & 0xf0f0f0f0u; };
    auto hi = [](uint32_t x) -> uint32_t { return x & 0xf0f0f0f0u; };
#pragma unroll 1
    for (int rb = 0; rb < n; rb += 16) {
        uint2 a0[kMaxK], a1[kMaxK], b[kMaxK], nx[kMaxK];
        load(rb + g, a0);
        load(rb + 8 + g, a1);
        load(g, nx);
        int sum[2] = {0, 0};
#pragma unroll 1
        for (int cb = 0; cb < nc; ++cb) {
#pragma unroll
            for (int Q = 0; Q < kMaxK; ++Q) b[Q] = nx[Q];
            if (cb + 1 < nc) load(8 * (cb + 1) + g, nx);
            int c[4] = {0, 0, 0, 0};
#pragma unroll
            for (int Q = 0; Q < kMaxK; ++Q) {
                if (Q < nk) {
                    mma_s8(c, lo(a0[Q].x), lo(a1[Q].x), hi(a0[Q].x), hi(a1[Q].x), lo(b[Q].x), hi(b[Q].x));
                    mma_s8(c, lo(a0[Q].y), lo(a1[Q].y), hi(a0[Q].y), hi(a1[Q].y), lo(b[Q].y), hi(b[Q].y));
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = rb + 8 * h + g, o = 8 * cb + 2 * t;
                const int d0 = r == o ? 0 : c[2 * h] >> 8, d1 = r == o + 1 ? 0 : c[2 * h + 1] >> 8;
                over = over || iabs(d0) > kByteMax || iabs(d1) > kByteMax;
                sum[h] += packed_abs(d0) + packed_abs(d1);
                p_sq += (long long)(d0 * d0 + d1 * d1);
                p_par += (d0 & 1) + (d1 & 1);
                if (r < n) {
                    if (halves) *reinterpret_cast<uint32_t*>(gp + (uint32_t)r * gst + 2u * (uint32_t)o) =
                        (uint32_t)(32768 + d0) | ((uint32_t)(32768 + d1) << 16);
                    else *reinterpret_cast<uint16_t*>(gp + (uint32_t)r * gst + (uint32_t)o) =
                        (uint16_t)((uint32_t)((128 + d0) & 255) | ((uint32_t)((128 + d1) & 255) << 8));
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            sum[h] += __shfl_xor_sync(FULL, sum[h], 1);
            sum[h] += __shfl_xor_sync(FULL, sum[h], 2);
            const int r = rb + 8 * h + g;
            if (t == 0 && r < n) {
                res[r] = sum[h];
                p_score += sum[h] & ((1 << kConfShift) - 1);
                p_conf += sum[h] >> kConfShift;
            }
        }
    }
    return __any_sync(FULL, !halves && over);
}

// Hybrid form: W as nibble pairs and the minority lists into the slot; G
// and the residuals from the arena when it holds them (XW_STATUS_GRAM: the
// totals are then the residuals' and the header's), else G built into it.
__device__ __forceinline__ bool build_hybrid(const Env& E, const XwJob* J, const uint8_t* rec, uint8_t* arena,
                                             uint32_t status0, int w, int lane, int& score0, int& conf0, int& par0,
                                             long long& sq0, bool& halves) {
    const int n = E.n, m = E.m, sparse = E.sparse;
    const uint32_t slot = E.slot, st = E.st, wbase = wbase_of<16>(slot, n);
    const int8_t* gw = reinterpret_cast<const int8_t*>(rec + J->off_w);
    int* res = reinterpret_cast<int*>(xw_smem + slot + Slot<16>::res);
    const bool cached = status0 & XW_STATUS_GRAM;
    int bad = 0;
    if (n > kHybridMaxOrder) return false;
    if (cached) {
        // the slot's W as the last launch left it (made from the record's bytes
        // again, and stored with a test on each byte, a launch of one iteration
        // of W(276,275) took 178 us and one of W(286,265) 379; 36 and 51 so)
        const uint4* src = reinterpret_cast<const uint4*>(arena + hybrid_arena(n).off_rows + 16u);
        const int chunks = (int)(hybrid_w_bytes(n) / 16u);
#pragma unroll 8
        for (int i = lane; i < chunks; i += 32) reinterpret_cast<uint4*>(xw_smem + wbase)[i] = __ldcg(src + i);
    }
    const bool whole = (n & 3) == 0;   // every word of the record is aligned and full
#pragma unroll 1
    for (int q = cached ? (int)st : lane; q < (int)st; q += 32) {
        const bool word = whole && 4 * q < n;
#pragma unroll 1
        for (int c0 = 0; c0 < n; c0 += 4) {
            uint32_t v[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int8_t* g = gw + (uint32_t)((c0 + k) * n + 4 * q);
                if (word && c0 + k < n) {
                    v[k] = *reinterpret_cast<const uint32_t*>(g);
                } else if (c0 + k < n) {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (4 * q + i < n) v[k] |= (uint32_t)(uint8_t)g[i] << (8 * i);
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (__vabs4(v[k]) & 0xfefefefeu) bad = 1;
                // bits 0, 8, 16, 24 to bits 24..27
                const uint32_t sup = ((v[k] & 0x01010101u) * 0x01020408u) >> 24,
                               neg = (((v[k] >> 7) & 0x01010101u) * 0x01020408u) >> 24;
                if (c0 + k < n) xw_smem[wbase + (uint32_t)(c0 + k) * st + (uint32_t)q] = (uint8_t)((sup & 15u) | ((neg & 15u) << 4));
            }
        }
    }
    const uint16_t* gmo = reinterpret_cast<const uint16_t*>(rec + J->off_mino);
    if (m == 0 && lane == 0 && (uint32_t)(2 * n * m) <= kHybridMino) E.mp[0] = 0;   // an empty list reads as column 0
    if (m > 0 && (status0 & XW_STATUS_INIT) && E.mp != gmo)
        for (int i = lane; i < n * m; i += 32) E.mp[i] = gmo[i];
    __syncwarp();
    int p_score = 0, p_conf = 0, p_par = 0;
    long long p_sq = 0;
    halves = false;
    if (cached) {
        halves = *reinterpret_cast<const uint32_t*>(arena + hybrid_arena(n).off_rows) != 0;
        const int* ares = reinterpret_cast<const int*>(arena);
        for (int o = lane; o < n; o += 32) {
            const int r = ares[o];
            res[o] = r;
            p_score += r & ((1 << kConfShift) - 1);
            p_conf += r >> kConfShift;
        }
    } else {
        uint8_t* rows = arena + hybrid_arena(n).off_rows;
        const uint32_t rst = hybrid_row_stride(n);
#pragma unroll 1
        for (int o = lane; o < n; o += 32) {
            int weight = 0, pos = 0;
#pragma unroll 1
            for (uint32_t q = 0; 16u * q < rst; ++q) {
                uint32_t sup = 0, w4[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const int c = 32 * (int)q + i;
                    if (c < n) {
                        const uint32_t v = w_at<16>(wbase, st, o, c) - 1u;
                        sup |= (v & 1u) << i;
                        w4[i >> 3] |= (v & 15u) << (4 * (i & 7));
                    }
                }
                *reinterpret_cast<uint4*>(rows + (uint32_t)o * rst + 16u * q) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                weight += __popc(sup);
                const int left = n - 32 * (int)q;
                if (m > 0 && !(status0 & XW_STATUS_INIT) && left > 0) {
                    uint32_t x = (sparse ? sup : ~sup) & (left >= 32 ? 0xffffffffu : (1u << left) - 1u);
                    while (x && pos < m) {
                        E.mp[o * m + pos] = (uint16_t)(32 * q + __ffs((int)x) - 1);
                        x &= x - 1;
                        ++pos;
                    }
                }
            }
            if (weight != w) bad = 1;
        }
        if (__any_sync(FULL, bad)) return false;
        __syncwarp();
#pragma unroll 1
        while (hybrid_gram(halves, E.gp, rows, res, n, lane, p_score, p_conf, p_par, p_sq)) {
            halves = true;
            p_score = p_conf = p_par = 0;
            p_sq = 0;
            __syncwarp();
        }
    }
    if (__any_sync(FULL, bad)) return false;
    score0 = __reduce_add_sync(FULL, p_score) / 2;
    conf0 = __reduce_add_sync(FULL, p_conf) / 2;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) p_sq += __shfl_xor_sync(FULL, p_sq, off);
    sq0 = p_sq / 2;
    par0 = __reduce_add_sync(FULL, p_par) / 2;
    __syncwarp();
    return true;
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
__device__ __forceinline__ bool load_replica(const AnnealArgs& a, uint32_t rid, uint32_t slot, int lane, uint64_t iters,
                                             Env& E, bool owner) {
    const unsigned gm = group_mask<GW>();
    uint8_t* rec = a.arena + a.rec_off[rid];
    RepHeader* H = reinterpret_cast<RepHeader*>(rec);
    XwJob* J = a.jobs + H->job;
    if (owner && *(volatile int32_t*)&J->done) return false;
    if (owner && a.stop_on_solve == 1 && *(volatile int32_t*)&J->solved) return false;
    const int obj_kind = GEN ? H->obj_kind : 0;
    if ((ONEZ && (J->m != 1 || J->sparse != 0)) || (!GEN && (H->obj_kind != 0 || J->move_set != 0))) {
        // a launch of a specialised kernel met a replica it does not cover
        if (lane == 0) H->err |= XW_ERR_KERNEL;
        return false;
    }
    make_env<WPL, GEN, GW, ONEZ>(E, J, slot, slot + Slot<WPL>::draws, lane, obj_kind);
    const int w = ONEZ ? E.n - 1 : J->w;
    const uint64_t it = H->it;
    if (J->budget_iters) {
        if (it >= J->budget_iters) return false;
        if (iters > J->budget_iters - it) iters = J->budget_iters - it;
    }
    const uint32_t status0 = H->status;
    int score0, conf0, par0;
    long long sq0;
    bool ok;
    bool halves = false, cached = false;   // hybrid form: G is in halfwords; the arena holds this W's G and residuals
    if constexpr (WPL == 16) {
        uint8_t* arena = a.gram + a.gram_off[rid];
        E.gp = arena + hybrid_arena(E.n).off_g;
        E.mp = (uint32_t)(2 * E.n * E.m) <= kHybridMino ? reinterpret_cast<uint16_t*>(xw_smem + E.mino)
                                                        : reinterpret_cast<uint16_t*>(rec + J->off_mino);
        cached = status0 & XW_STATUS_GRAM;
        ok = build_hybrid(E, J, rec, arena, status0, w, lane, score0, conf0, par0, sq0, halves);
    } else if constexpr (WPL == 8) ok = build_wide(E, J, rec, status0, w, lane, score0, conf0, par0, sq0);
    else ok = build_packed<WPL, GW>(E, J, rec, status0, w, lane, score0, conf0, par0, sq0);
    if (!ok) {
        if (lane == 0 && owner) H->err |= XW_ERR_MINORITY;
        return false;
    }

    const int64_t obj0 = cached && obj_kind != 0 ? H->obj_total : obj_kind == 1 ? sq0 : obj_kind == 2 ? par0 : score0;
    const bool init = status0 & XW_STATUS_INIT;
    if (init && (H->score != score0 || H->conflicts != conf0 || H->obj_total != obj0)) {
        if (lane == 0 && owner) H->err |= XW_ERR_SCORE;
        return false;
    }
    if (lane == 0) {
        Con c;
        c.thr_target = J->thr_target;
        c.thr_dbl = GEN && J->move_set == 1 ? 0 : J->thr_double;
        c.thr_sign = J->thr_sign;
        c.thr_swsign = J->thr_swsign;
        c.k0 = J->key0;
        c.k1 = J->key1;
        c.stream = H->stream;
        c.cs = J->candidate_samples;
#pragma unroll
        for (uint32_t r = 0; r < 5; ++r)
            c.keys[r] = make_uint4(c.k0 + 2 * r * 0x9E3779B9u, c.k1 + 2 * r * 0xBB67AE85u,
                                   c.k0 + (2 * r + 1) * 0x9E3779B9u, c.k1 + (2 * r + 1) * 0xBB67AE85u);
        c.it0 = it;
        c.thr_greedy = J->thr_greedy;
        auto coin = [](uint64_t t) -> uint32_t { return t > 0xffffffffull ? 0xffffffffu : (uint32_t)t; };
        c.coins = make_uint4(coin(c.thr_target), coin(c.thr_dbl), coin(c.thr_sign), coin(c.thr_swsign));
        c.T = H->temperature;
        c.best = make_int4(score0, conf0, init ? H->best_score : score0, init ? H->best_conflicts : conf0);
        c.acc = make_int4((int)(uint32_t)obj0, (int)(obj0 >> 32), init ? (int)H->accepted : 0,
                          init ? (int)H->accepted_rows : 0);
        // (a tempering replica's count of calls without improvement goes on
        // for as long as it runs, and wraps)
        c.mb = init ? (int32_t)(0u - (uint32_t)H->msi) : 0;
        c.cb = init ? -H->cool_ctr : 0;
        c.mpc = J->moves_per_cool;
        c.stuck = J->stuck_threshold;
        c.fixed = J->tempering;
        c.k_end = xw_launch_calls(iters);
        c.jn = init ? -1 : 0;
        c.owner = owner ? 1 : 0;
        c.halves = halves ? 1 : 0;
        c.rid = rid;
        *con_of<WPL>(slot) = c;
    }
    __syncwarp(gm);
    build_thresholds<GW>(reinterpret_cast<uint32_t*>(xw_smem + slot + Slot<WPL>::thr), H->temperature, lane);
    return true;
}

// Writes the replica's W, minority lists and scalar state back to its
// record after `k` calls, with `evals` candidates evaluated, `evals2` of
// them changing two rows.
template <int WPL, int GW>
__device__ __forceinline__ void store_replica(const AnnealArgs& a, const Env& E, int k, uint64_t evals, uint32_t evals2,
                                              int lane) {
    const unsigned gm = group_mask<GW>();
    __syncwarp(gm);
    const Con* con = con_of<WPL>(E.slot);
    uint8_t* rec = a.arena + a.rec_off[con->rid];
    RepHeader* H = reinterpret_cast<RepHeader*>(rec);
    const XwJob* J = a.jobs + H->job;
    const uint32_t wbase = wbase_of<WPL>(E.slot, E.n);
    if (con->jn >= 0) save_best<WPL, GW>(rec, J, E, con->jn, lane);
    save_w<WPL, GW>(reinterpret_cast<int8_t*>(rec + J->off_w), wbase, E.st, E.n, lane);
    if constexpr (WPL == 16) {
        uint16_t* gmo = reinterpret_cast<uint16_t*>(rec + J->off_mino);
        if (gmo != E.mp)
            for (int i = lane; i < E.n * E.m; i += GW) gmo[i] = E.mp[i];
        int* res = reinterpret_cast<int*>(a.gram + a.gram_off[con->rid]);
        if (lane == 0)
            *reinterpret_cast<uint32_t*>(a.gram + a.gram_off[con->rid] + hybrid_arena(E.n).off_rows) = con->halves ? 1u : 0u;
        for (int o = lane; o < E.n; o += GW) res[o] = reinterpret_cast<const int*>(xw_smem + E.slot + Slot<WPL>::res)[o];
        uint4* keep = reinterpret_cast<uint4*>(a.gram + a.gram_off[con->rid] + hybrid_arena(E.n).off_rows + 16u);
        for (int i = lane; i < (int)(hybrid_w_bytes(E.n) / 16u); i += GW)
            keep[i] = *reinterpret_cast<const uint4*>(xw_smem + wbase + 16u * (uint32_t)i);
    } else {
        uint8_t* gmo = rec + J->off_mino;
        for (uint32_t i = lane; i < (uint32_t)(E.n * E.m); i += GW) gmo[i] = xw_smem[E.mino + i];
    }
    if (lane == 0) {
        const bool init = H->status & XW_STATUS_INIT;
        H->it = con->it0 + (uint64_t)k;
        H->moves = (init ? H->moves : 0) + (uint64_t)k;
        H->cand_evals = (init ? H->cand_evals : 0) + evals;
        H->accepted = (uint32_t)con->acc.z;
        H->accepted_rows = (uint32_t)con->acc.w;
        H->two_row_evals = (init ? H->two_row_evals : 0) + evals2;
        H->score = con->best.x;
        H->conflicts = con->best.y;
        H->best_score = con->best.z;
        H->best_conflicts = con->best.w;
        H->obj_total = (int64_t)(((uint64_t)(uint32_t)con->acc.y << 32) | (uint32_t)con->acc.x);
        H->temperature = con->T;
        H->msi = (int32_t)((uint32_t)k - (uint32_t)con->mb);
        H->cool_ctr = J->tempering ? -con->cb : k - con->cb;   // tempering leaves it alone
        H->status = H->status | XW_STATUS_INIT | (WPL == 16 ? XW_STATUS_GRAM : 0u) | (con->best.z == 0 ? XW_STATUS_SOLVED : 0u);
    }
    __syncwarp(gm);
}

// Commits the accepted move `mv` of call k (iteration it0 + k - 1; k counts
// it) with deltas `acc` and `prim`: the state, best tracking and the job's
// solve flag.  True when the best improved.
template <int WPL, bool GEN, int GW, bool ONEZ>
__device__ __forceinline__ bool accept_move(const AnnealArgs& a, const Env& E, const Move& mv, int acc, int prim, int k,
                                            int lane) {
    const unsigned gm = group_mask<GW>();
    Con* con = con_of<WPL>(E.slot);
    const int dc = (acc + 2048) >> 12;
    int4 b = con->best, t = con->acc;
    const int jn = con->jn;
    b.x += acc - dc * 4096;
    b.y += dc;
    const bool improved = b.x < b.z || (b.x == b.z && b.y < b.w);
    if (jn == kJournal && !improved && con->owner) {
        uint8_t* rec = a.arena + a.rec_off[con->rid];
        save_best<WPL, GW>(rec, a.jobs + reinterpret_cast<RepHeader*>(rec)->job, E, jn, lane);
    }
    if constexpr (WPL == 16) commit_hybrid(E, mv, acc, lane);
    else if constexpr (WPL == 8) commit_wide<ONEZ>(E, mv, acc, lane);
    else commit<WPL, GW, ONEZ>(E, mv, acc, lane);
    if (lane == 0) {
        const long long o = (long long)(((uint64_t)(uint32_t)t.y << 32) | (uint32_t)t.x) + prim;
        t.x = (int)(uint32_t)o;
        t.y = (int)(o >> 32);
        t.z += 1;
        t.w += (mv.rc & 255u) != ((mv.rc >> 8) & 255u) || ((mv.ax >> 26) & 1u) != ((mv.ax >> 27) & 1u) ? 2 : 1;
        con->acc = t;
        if (improved) {
            b.z = b.x;
            b.w = b.y;
            con->mb = k;
            if (b.x == 0 && con->owner) {
                RepHeader* H = reinterpret_cast<RepHeader*>(a.arena + a.rec_off[con->rid]);
                XwJob* J = a.jobs + H->job;
                H->solve_it = con->it0 + (uint64_t)(k - 1);
                H->solve_ns = globaltimer();
                if (atomicCAS(&J->solved, 0, 1) == 0) {
                    J->solved_replica = (int32_t)H->stream;
                    J->solved_it = H->solve_it;
                    J->solve_ns = H->solve_ns;
                }
            }
        }
        con->best = b;
        if (improved) {
            con->jn = 0;
        } else if (jn >= 0) {
            if (jn < kJournal)
                *reinterpret_cast<uint2*>(xw_smem + E.slot + Slot<WPL>::jrn + 8u * (uint32_t)jn) =
                    make_uint2(mv.rc, (mv.cf & 15u) | ((mv.cf >> 4) & 0xf0u) | ((mv.cf >> 8) & 0xf00u) |
                                          ((mv.cf >> 12) & 0xf000u) | (((mv.ax >> 26) & 15u) << 16));
            con->jn = jn < kJournal ? jn + 1 : -1;
        }
    }
    __syncwarp(gm);
    return improved;
}

// Calls that can be made after call k before the temperature changes or
// the replica's calls end: the first k at which temperature_step has
// something to do.
__device__ __forceinline__ int next_event(const Con* con) {
    if (con->fixed) return con->k_end;
    const long long e = min((long long)con->cb + con->mpc, (long long)con->mb + con->stuck);
    return (int)min(e, (long long)con->k_end);
}

// Cooling and reheat after call k (xweigh_cuda.cu:1087-1129); neither under
// tempering.
template <int WPL, int GW>
__device__ __forceinline__ void temperature_step(const AnnealArgs& a, uint32_t slot, int k, int lane) {
    const unsigned gm = group_mask<GW>();
    Con* con = con_of<WPL>(slot);
    if (con->fixed) return;
    const bool cool = (long long)k - con->cb >= con->mpc, heat = (long long)k - con->mb >= con->stuck;
    if (!cool && !heat) return;
    const RepHeader* H = reinterpret_cast<const RepHeader*>(a.arena + a.rec_off[con->rid]);
    const XwJob* J = a.jobs + H->job;
    const double T0 = con->T, t_min = J->t_min;
    double T = T0;
    if (cool) {
        T = __dmul_rn(T, J->cooling);
        if (T < t_min) T = t_min;
    }
    if (heat) {
        T = __dmul_rn(H->reheat_temperature, J->reheat);
        if (T < t_min) T = t_min;
    }
    __syncwarp(gm);
    if (lane == 0) {
        if (cool) con->cb = k;
        if (heat) con->mb = k;
        con->T = T;
    }
    if (T != T0) build_thresholds<GW>(reinterpret_cast<uint32_t*>(xw_smem + slot + Slot<WPL>::thr), T, lane);
    __syncwarp(gm);
}

}  // namespace
}  // namespace xw
