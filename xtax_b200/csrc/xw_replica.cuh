// xw_replica.cuh -- the replica loop on packed rows (xw_packed.cuh) and the
// kernel of one replica per warp or half-warp, shared by the files that
// instantiate it: xw_anneal.cu (orders up to 32), xw_anneal_wide.cu (orders
// above), xw_spec_lean.cu and xw_spec_general.cu (the latency mode).
//
// Each of these files is a module of its own, which a process loads when it
// first uses a kernel of it; line tables are most of its size.  The first
// batch of a process, from its creation to its results, ms, with one module
// of 25 MB / with these: W(12,11) alone 36 / 15, 1000 replicas of W(26,25)
// 40 / 17, W(100,50) 57 / 36, W(276,275) 49 / 29.
#pragma once

#include <cuda_runtime.h>

#define XW_EDGE_INLINE
#include "xw_device.cuh"
#include "xw_kernels.h"
#include "xw_packed.cuh"

namespace xw {

namespace {

// Position of a replica's loop.
struct Walk {
    int k;               // calls made
    int wpos;            // next iteration of the window of move-level draws
    uint32_t wmask;      // bit j: iteration j of the window has several candidates
    uint32_t multis;     // iterations of several candidates
    uint32_t two_l;      // two-row candidates of this lane's group
};

// One step of a replica, at most to call k_lim: returns whether a move was
// accepted; `improved`: it is the best yet.
//
// An iteration proposes one candidate or, with the job's greedy
// probability, candidate_samples of them.  A step gives its four candidate
// groups either the candidates of one iteration or, in a run of
// one-candidate iterations, the next up to four iterations of the run:
// their draws and the kind of each are known ahead (counter-based), and
// while no move is accepted they see the same state.  The first accepted
// one is committed; the iterations after it are proposed again.  The
// trajectory is that of one iteration at a time.  (Acceptance is 11% on the
// W(26,25) ladder: 0.85 steps an iteration.)
template <int WPL, bool GEN, int GW, bool ONEZ>
__device__ __forceinline__ bool step(const AnnealArgs& a, const Env& E, Walk& w, int k_lim, int lane, bool& improved) {
    constexpr int LPC = GW / 4;
    constexpr int kWin = GW;   // iterations whose move-level draws are computed at once
    const unsigned gm = group_mask<GW>();
    const int wl0 = GW == 32 ? 0 : (int)(threadIdx.x & 16u);
    const Con* con = con_of<WPL>(E.slot);
    const int g = lane / LPC;
    const uint32_t win = E.slot + Slot<WPL>::win;
    if (w.wpos >= kWin) {
        const uint4 b = draw_block(0u, con->it0 + (uint64_t)w.k + (uint64_t)lane, con->stream, con->k0, con->k1);
        w.wmask = __ballot_sync(gm, (uint64_t)b.x < con->thr_greedy) >> wl0;
        *reinterpret_cast<uint32_t*>(xw_smem + win + 4u * (uint32_t)lane) = b.y;
        w.wpos = 0;
        __syncwarp(gm);
    }
    const uint32_t rem = w.wmask >> w.wpos;
    const bool multi = rem & 1u;
    const uint64_t it = con->it0 + (uint64_t)w.k;
    bool accept;
    int used = 1, acc, prim;
    Move mv;
    w.multis += rem & 1u;
    if (multi && con->cs > 4) {
        const Winner c = choose_many<WPL, GEN, GW, ONEZ>(E, it, con->cs, lane);
        mv = c.mv;
        acc = c.acc;
        prim = c.prim;
        if (lane == 0) w.two_l += (uint32_t)c.two;
        accept = accepts<WPL>(E.slot, prim, lds32(win + 4u * (uint32_t)w.wpos));
    } else {
        const int run = multi ? con->cs : min(min(__ffs((int)(rem | 16u)) - 1, kWin - w.wpos), k_lim - w.k);
        const bool act = g < run;
        fill_draws<GW>(E, con, it, 0, multi, lane);
        __syncwarp(gm);
        const Cand q = candidate<WPL, GEN, GW, ONEZ>(E, it, multi ? 0 : g, multi ? g : 0, act, lane);
        const bool ok = accepts<WPL>(E.slot, q.prim, lds32(win + 4u * (uint32_t)(w.wpos + (multi ? 0 : g))));
        const uint32_t oks = __ballot_sync(gm, act && ok) >> wl0;
        // the best candidate, or the first accepted iteration of a run
        uint32_t A, B;
        best_keys(GEN && E.obj_kind != 0, q, act && (multi || ok), g, !multi, gm, A, B);
        const int src = (int)(B & 3u) * LPC;
        accept = (oks >> src) & 1u;   // (a run without one: group 3, whose bit is clear)
        if (!multi) used = accept ? (int)(B & 3u) + 1 : run;
        w.two_l += q.R2 != q.R1 && (multi ? act : g < used) ? 1u : 0u;
        if (accept) {
            mv = move_of(pack_move<WPL>(q), wl0 + src, gm);
            acc = __shfl_sync(gm, q.acc, wl0 + src);
            prim = __shfl_sync(gm, q.prim, wl0 + src);
        }
    }
    w.k += used;
    w.wpos += used;
    improved = accept && accept_move<WPL, GEN, GW, ONEZ>(a, E, mv, acc, prim, w.k, lane);
    return accept;
}

// The one-warp (or half-warp) replica loop.
template <int WPL, bool GEN, int GW, bool ONEZ>
__device__ __forceinline__ void run_replica(const AnnealArgs& a, uint32_t rid, uint32_t slot, int lane,
                                            uint64_t iters) {
    constexpr int LPC = GW / 4;
    Env E;
    if (!load_replica<WPL, GEN, GW, ONEZ>(a, rid, slot, lane, iters, E, true)) return;
    auto job = [&]() -> XwJob* { return a.jobs + reinterpret_cast<const RepHeader*>(a.arena + a.rec_off[rid])->job; };
    // stop rules: 1, every replica of the job stops soon after any solve;
    // 2, a replica stops at its own solve only, so that each replica's
    // trajectory is independent of how the launches are scheduled
    auto stops = [&](const Con* con, int k) -> bool {
        if (k >= con->k_end) return true;
        if (a.stop_on_solve && con->best.z == 0) return true;
        return a.stop_on_solve == 1 && (k & 63) == 63 && *(volatile int32_t*)&job()->solved;
    };
    // the next k at which something besides moves happens
    auto event = [&](const Con* con, int k) -> int {
        int e = xw_event_after(next_event(con), k);
        if (a.stop_on_solve == 1) e = min(e, xw_event_after(0, k) | 63);   // calls 63, 127, ...
        return e;
    };
    Walk w{0, GW, 0u, 0u, 0u};
    int k_evt = event(con_of<WPL>(slot), 0);
    bool live = !stops(con_of<WPL>(slot), 0);
#pragma unroll 1
    while (live) {
        // values derived from these are computed where they are used: held
        // across the loop they cost more in spilled registers
        asm volatile("" : "+r"(E.slot), "+r"(lane));
        const Con* con = con_of<WPL>(E.slot);
        bool improved;
        step<WPL, GEN, GW, ONEZ>(a, E, w, k_evt, lane, improved);
        // an improvement puts the reheat off (an event due now still comes)
        if (improved && w.k < k_evt) k_evt = a.stop_on_solve && con->best.z == 0 ? w.k : event(con, w.k);
        if (w.k >= k_evt) {
            temperature_step<WPL, GW>(a, E.slot, w.k, lane);
            live = !stops(con, w.k);
            k_evt = event(con, w.k);
        }
    }
    const uint64_t evals =
        (uint64_t)((uint32_t)w.k - w.multis) + (uint64_t)w.multis * (uint64_t)con_of<WPL>(E.slot)->cs;
    const uint32_t evals2 = __reduce_add_sync(group_mask<GW>(), (lane & (LPC - 1)) == 0 ? w.two_l : 0u);
    store_replica<WPL, GW>(a, E, w.k, evals, evals2, lane);
}

// Register budget per thread; it sets how many replica warps an SM holds.
// An SM's registers are split between its four schedulers (16384 each): 80
// registers per thread give 6 warps per scheduler, 96 give 5, 112 and 128
// give 4.  The one-row kernels take the smallest budget next to free of spills:
// measured on B200 (W(26,25) ladder, 4096 replicas, 10^4 iterations) 19.5
// ms at 96 registers, 20.8 at 112, 21.7 at 80 (180 bytes of spills a
// thread), 24.1 at 72; the general kernel (W(24,23), 2368 replicas, 4096
// iterations) 9.7 ms at 112, 9.9 at 96, 10.3 at 80.
#ifndef XW_ANNEAL_MAXNREG
#define XW_ANNEAL_MAXNREG 128
#endif
#ifndef XW_ANNEAL_MAXNREG_LEAN1
#define XW_ANNEAL_MAXNREG_LEAN1 96
#endif
#ifndef XW_ANNEAL_MAXNREG_GEN1
#define XW_ANNEAL_MAXNREG_GEN1 112
#endif
#ifndef XW_ANNEAL_MAXNREG_PAIR
#define XW_ANNEAL_MAXNREG_PAIR 96
#endif
#ifndef XW_ANNEAL_MAXNREG_WIDE
#define XW_ANNEAL_MAXNREG_WIDE 208
#endif
constexpr int anneal_maxnreg(int opl, bool general, int gw) {
    return opl == 8 ? XW_ANNEAL_MAXNREG_WIDE
           : gw == 16 ? XW_ANNEAL_MAXNREG_PAIR
                    : opl == 1 ? (general ? XW_ANNEAL_MAXNREG_GEN1 : XW_ANNEAL_MAXNREG_LEAN1) : XW_ANNEAL_MAXNREG;
}

// Each lane group (the warp, or each half of it) takes work items from the
// launch's counter on its own: a replica (all of its launch iterations) or
// one chunk of them.
template <int OPL, bool GEN, int GW, bool ONEZ = false>
__global__ void __maxnreg__(anneal_maxnreg(OPL, GEN, GW)) anneal_kernel(AnnealArgs a) {
    const int lane = threadIdx.x & (GW - 1);
    const int group = threadIdx.x / GW;
    const unsigned gm = group_mask<GW>();
    const uint32_t slot = (uint32_t)group * a.slot_bytes;
    const uint64_t total = (uint64_t)a.n_items * a.chunks;
    for (;;) {
        uint32_t item = 0;
        if (lane == 0) item = atomicAdd(a.counter, 1u);
        item = __shfl_sync(gm, item, 0, GW);
        if (item >= total) break;
        // chunk c of the replica's launch iterations (one chunk: all of them)
        const uint32_t c = a.chunks == 1 ? 0u : item / a.n_items;
        const uint32_t rid = a.items[item - c * a.n_items];
        const uint64_t lo = a.iters * c / a.chunks, hi = a.iters * (c + 1) / a.chunks;
        RepHeader* H = reinterpret_cast<RepHeader*>(a.arena + a.rec_off[rid]);
        const bool chunked = a.chunks > 1;
        const bool ok = !chunked || chunk_begin(a.chunk_done + rid, c, a.chunk_wait_ns, &H->err, lane, gm);
        if (ok) {
            run_replica<OPL, GEN, GW, ONEZ>(a, rid, slot, lane, hi - lo);
        }
        if (chunked) chunk_end(a.chunk_done + rid, c, ok, lane, gm);
    }
}

}  // namespace

}  // namespace xw
