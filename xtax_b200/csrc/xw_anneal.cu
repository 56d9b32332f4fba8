// xw_anneal.cu -- the population annealing kernel for weighing matrices.
//
// One warp (or a half-warp) owns one replica at a time, its state in the
// warp's shared-memory slot; the whole iteration is warp-synchronous: no
// __syncthreads, no block-wide reductions.  The iteration itself is in
// xw_packed.cuh: rows of W and G packed into words, bytes of G up to order
// 128, halfwords above.
//
// Per iteration (the semantics of the reference kernel anneal_kernel,
// src/xweigh_cuda.cu:988-1130, with cuRAND replaced by counter-based Philox):
//   A  every lane computes one Philox block of this iteration's draws
//      (move-level block + the common blocks of the first candidates) into
//      shared memory;
//   C  hot-row tournaments (xweigh_cuda.cu:291-300), 8 samples per candidate;
//   D  proposals (propose_move, xweigh_cuda.cu:423-447);
//   E  candidate evaluation, the first best kept (device_better_evaluation,
//      xweigh_cuda.cu:227-244);
//   F  Metropolis on the replica's objective with the integer draw and the
//      deterministic acceptance exponential;
//   G  the commit (commit_*, xweigh_cuda.cu:607-877);
//   H  best tracking, cooling and reheat (xweigh_cuda.cu:1087-1129).
//
// Work distribution is persistent: each warp takes replica ids from a
// global counter until the launch's item list is exhausted, so replicas of
// different orders and weights share one launch.
#include <cuda_runtime.h>

#include <algorithm>

#include <cooperative_groups.h>

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

// Latency mode: one replica per CTA of K warps, speculating K iterations at
// a time.  Warp k computes iteration it + k (phases A-E) against the
// replica's current state, each with its own draw buffer: the draws of an
// iteration depend only on its number, and its proposals and deltas only on
// the state, which no iteration changes before one is accepted.  Warp 0
// then takes the iterations in order through phases F-H until the first
// accepted one, commits it, and discards the iterations after it, whose
// proposals read the state it changed; the next round starts after the
// accepted iteration.  The trajectory is the one-warp kernel's, move for
// move; a round advances by the run of rejections up to the next accept
// (about 2-4 iterations at the acceptance rates of cooling runs) in about
// the time of one iteration, so a lone search runs that much faster.

//
// Where moves are accepted every iteration or two a round advances no
// further than one step of the one-warp loop and takes longer (2000
// iterations of W(12,11) with its hottest replica accepting all: 3.15 ms in
// the one-warp loop, 4.1 with 2 warps, 6.1 with 16, 8.2 with 64 on four SMs).
// So warp 0 watches the advance: below kSoloAdvance iterations a round it
// goes on alone, step by step, until accepts are rare enough again (in a
// cluster every CTA's warp 0 makes the same steps on its copy).

// Per-warp results and the round's control word, after the slot's own
// (warp 0's) structures and the other warps' draw buffers.
struct SpecOut {
    Move mv;
    int32_t dsc, prim;        // score change + 4096 x conflict change; objective change
    uint32_t u;
    uint32_t evals, evals2;   // candidates evaluated; those changing two rows
    int32_t acc;              // the Metropolis outcome at the round's starting temperature
};
struct SpecCtl {
    int32_t k;          // calls made before the round
    int32_t count;      // iterations of the round (0: the replica stops)
};

// Per round buffer (two, used in turn): the outcomes of all the round's
// warps (K per CTA, CL CTAs), and the job's solved flag as the cluster's
// owner read it.
struct SpecLayout {
    uint32_t off_extra, off_out, out_stride, off_flag, off_ctl, bytes;
};

// the latency-mode regions after a slot of `slot_bytes` (the one-warp
// layout of the largest of a launch's replicas), for K warps per CTA and
// CL CTAs per replica
__host__ __device__ inline SpecLayout spec_layout(uint32_t slot_bytes, int K, int CL) {
    SpecLayout S;
    S.off_extra = xw_pad16(slot_bytes);
    S.off_out = S.off_extra + (uint32_t)(K - 1) * 512u;
    S.out_stride = xw_pad16((uint32_t)(K * CL) * (uint32_t)sizeof(SpecOut));
    S.off_flag = S.off_out + 2u * S.out_stride;
    S.off_ctl = xw_pad16(S.off_flag + 2u * 4u);
    S.bytes = S.off_ctl + (uint32_t)sizeof(SpecCtl);
    return S;
}

// The replica loop of a CTA of the latency mode.  With CL > 1 the replica
// runs on a cluster of CL CTAs (on CL SMs): every CTA loads its own copy,
// the cluster's warps speculate CL * K iterations, every warp writes its
// outcome into every CTA's round buffer (distributed shared memory), and
// after a cluster barrier each CTA's warp 0 makes the same walk and the
// same commit on its own copy, so the copies stay identical; only rank 0
// writes the record.  Everything that steers the walk is either the
// CTAs' identical state or read by rank 0 alone and exchanged (whether
// the replica runs at all, and the job's solved flag each round), so the
// CTAs take the same branches and meet at every barrier.
template <int WPL, bool GEN, int CL, bool ONEZ>
__device__ void run_replica_spec(const AnnealArgs& a, uint32_t rid, int warp, int K, int lane) {
    namespace cg = cooperative_groups;
    const int rank = CL > 1 ? (int)cg::this_cluster().block_rank() : 0;
    const bool owner = rank == 0;
    const RepHeader* H = reinterpret_cast<const RepHeader*>(a.arena + a.rec_off[rid]);
    XwJob* J = a.jobs + H->job;
    const SpecLayout L = spec_layout(packed_slot_bytes(J->n, J->m, WPL), K, CL);
    SpecCtl* ctl = reinterpret_cast<SpecCtl*>(xw_smem + L.off_ctl);
    const Con* con = con_of<WPL>(0u);
    Env E;
    bool ok = false;
    const int KT = K * CL;
    int k = 0, k_evt = 0, k_end = 0;
    // a round's cost in steps of the one-warp loop, in tenths (measured)
    const int cost10 = CL > 1 ? 26 : 12 + K / 2;
    int rounds = 0, round_k = 0;   // rounds since the last look, and k then
    uint64_t evals = 0;
    uint32_t evals2 = 0;
    // warp 0 loads the replica; the round size goes to the others through
    // shared memory
    if (warp == 0) {
        ok = load_replica<WPL, GEN, 32, ONEZ>(a, rid, 0u, lane, a.iters, E, owner);
        if (ok) {
            k_evt = xw_event_after(next_event(con), 0);
            k_end = con->k_end;
        }
        if (lane == 0 && owner) {
            SpecCtl c;
            c.k = 0;
            c.count = !ok || (a.stop_on_solve && con->best.z == 0) ? 0 : min(k_end, KT);
            *ctl = c;
            if constexpr (CL > 1) {
                for (int q = 1; q < CL; ++q) *cg::this_cluster().map_shared_rank(ctl, q) = c;
            }
        }
    }
    if constexpr (CL > 1) cg::this_cluster().sync();
    else __syncthreads();
    if (ctl->count == 0) {
        // nothing to run: the loaded replica's record still gets its
        // rebuilt state, as the one-warp kernel writes it
        if (warp == 0 && ok && owner) store_replica<WPL, 32>(a, E, 0, 0, 0, lane);
        return;
    }
    // every warp: the replica's structures (read-only until warp 0 commits)
    // and its own draw buffer
    if (warp != 0)
        make_env<WPL, 32, ONEZ>(E, J, 0u, L.off_extra + (uint32_t)(warp - 1) * 512u, lane, GEN ? H->obj_kind : 0);

    const int g = rank * K + warp;   // this warp's iteration within the round
#pragma unroll 1
    for (int round = 0;; ++round) {
        const int buf = round & 1;
        SpecOut* outs = reinterpret_cast<SpecOut*>(xw_smem + L.off_out + (uint32_t)buf * L.out_stride);
        int32_t* flag = reinterpret_cast<int32_t*>(xw_smem + L.off_flag) + buf;
        const int cnt = ctl->count;
        if (g < cnt) {
            const uint64_t it = con->it0 + (uint64_t)(ctl->k + g);
            fill_draws<32, true>(E, con, it, 0, true, lane);
            __syncwarp();
            const uint64_t mblk = lds64(E.draws + 24u * 16u);
            const int count = (uint64_t)(uint32_t)mblk < con->thr_greedy ? con->cs : 1;
            SpecOut o;
            o.u = (uint32_t)(mblk >> 32);
            o.evals = (uint32_t)count;
            if (count > 4) {
                const Winner w = choose_many<WPL, GEN, 32, ONEZ>(E, it, count, lane);
                o.mv = w.mv;
                o.dsc = w.acc;
                o.prim = w.prim;
                o.evals2 = (uint32_t)w.two;
            } else {
                const int c = lane >> 3;
                const bool act = c < count;
                const Cand q = candidate<WPL, GEN, 32, ONEZ>(E, it, 0, c, act, lane);
                uint32_t A, B = 0;
                if (count > 1) best_keys(GEN && E.obj_kind != 0, q, act, c, false, FULL, A, B);
                const int src = (int)(B & 3u) * 8;
                o.mv = move_of(pack_move<WPL>(q), src, FULL);
                o.dsc = __shfl_sync(FULL, q.acc, src);
                o.prim = __shfl_sync(FULL, q.prim, src);
                o.evals2 = (uint32_t)__popc(__ballot_sync(FULL, act && q.R2 != q.R1 && (lane & 7) == 0));
            }
            // the Metropolis test at the round's starting temperature: the
            // one warp 0 would make if no cooling or reheat step falls
            // between the round's start and this iteration
            o.acc = accepts<WPL>(0u, o.prim, o.u) ? 1 : 0;
            if (lane == 0) {
                outs[g] = o;
                if constexpr (CL > 1) {
                    for (int q = 0; q < CL; ++q)
                        if (q != rank) cg::this_cluster().map_shared_rank(outs, q)[g] = o;
                }
            }
        }
        if constexpr (CL > 1) {
            if (owner && warp == 0 && lane == 0) {
                const int32_t sv = a.stop_on_solve == 1 ? *(volatile int32_t*)&J->solved : 0;
                for (int q = 0; q < CL; ++q) *cg::this_cluster().map_shared_rank(flag, q) = sv;
            }
            cg::this_cluster().sync();
        } else {
            __syncthreads();
        }
        if (warp == 0) {
            // Iterations in order until the first accepted move.  Fast path:
            // the rejected calls before it change only counters unless one
            // of them reaches a cooling or reheat step, so when none can,
            // they are counted in bulk and only the accepted move is
            // committed.  Otherwise the ordered walk.
            // The job's solved flag: read here on one CTA, as the owner read
            // it this round on a cluster.
            auto solved = [&]() -> bool {
                if constexpr (CL > 1) return *flag != 0;
                else return *(volatile int32_t*)&J->solved != 0;
            };
            // call k has been made; its temperature step
            auto after_call = [&]() {
                if (k >= k_evt) {
                    temperature_step<WPL, 32>(a, 0u, k, lane);
                    k_evt = xw_event_after(next_event(con), k);
                }
            };
            auto commit_of = [&](int q) {
                if (accept_move<WPL, GEN, 32, ONEZ>(a, E, outs[q].mv, outs[q].dsc, outs[q].prim, k, lane) && k < k_evt)
                    k_evt = xw_event_after(next_event(con), k);
            };
            // lane l looks at iterations l and 32 + l (up to 64 iterations a
            // round, on a cluster of four)
            const bool l0 = lane < cnt, l1 = 32 + lane < cnt;
            const uint64_t acc_m = (uint64_t)__ballot_sync(FULL, l0 && outs[l0 ? lane : 0].acc != 0) |
                                   ((uint64_t)__ballot_sync(FULL, l1 && outs[l1 ? 32 + lane : 0].acc != 0) << 32);
            const int ja = acc_m ? __ffsll((long long)acc_m) - 1 : -1;
            const int jend = ja >= 0 ? ja + 1 : cnt;
            const int rejects = ja >= 0 ? jend - 1 : jend;
            bool fast = rejects < k_evt - k;
            // a check of the job's solved flag (every 64th iteration) that
            // falls in the span and finds it set: take the span in order
            if (fast && a.stop_on_solve == 1 && (k | 63) < k + jend && solved()) fast = false;
            bool stop = false;
            if (fast) {
                const bool in0 = lane < jend, in1 = 32 + lane < jend;
                const uint32_t ev = __reduce_add_sync(
                    FULL, (in0 ? outs[lane].evals + (outs[lane].evals2 << 16) : 0u) +
                              (in1 ? outs[32 + lane].evals + (outs[32 + lane].evals2 << 16) : 0u));
                evals += ev & 0xffffu;
                evals2 += ev >> 16;
                k += jend;
                if (ja >= 0) commit_of(ja);
                after_call();
            } else {
#pragma unroll 1
                for (int j = 0; j < cnt; ++j) {
                    if (a.stop_on_solve == 1 && (k & 63) == 63 && solved()) {
                        stop = true;
                        break;
                    }
                    evals += outs[j].evals;
                    evals2 += outs[j].evals2;
                    const bool accept = accepts<WPL>(0u, outs[j].prim, outs[j].u);
                    ++k;
                    if (accept) commit_of(j);
                    after_call();
                    if (accept) break;
                }
            }
            if (a.stop_on_solve && con->best.z == 0) stop = true;
            // alone from here?  (a step of the one-warp loop makes 1.1
            // iterations or more)
            ++rounds;
            bool solo = false;
            if (rounds >= 8) {
                solo = (k - round_k) * 100 < rounds * cost10 * 11;
                rounds = 0;
                round_k = k;
            }
            if (solo && !stop) {
                Walk w{k, 32, 0u, 0u, 0u};
                // the job's solved flag is looked at between rounds only
                const int k_poll = a.stop_on_solve == 1 ? ((k | 63) == k ? k : k | 63) : k_end;
                while (solo) {
                    const int k1 = min(xw_calls_to(w.k, 64, k_end), k_poll);
                    int steps = 0, accs = 0;
                    while (w.k < k1) {
                        bool improved;
                        accs += step<WPL, GEN, 32, ONEZ>(a, E, w, min(k_evt, k1), lane, improved) ? 1 : 0;
                        ++steps;
                        if (improved && w.k < k_evt) k_evt = xw_event_after(next_event(con), w.k);
                        if (w.k >= k_evt) {
                            temperature_step<WPL, 32>(a, 0u, w.k, lane);
                            k_evt = xw_event_after(next_event(con), w.k);
                        }
                        if (a.stop_on_solve && con->best.z == 0) {
                            stop = true;
                            break;
                        }
                    }
                    solo = !stop && steps > 0 && w.k < k_poll && w.k < k_end && steps * 10 < accs * cost10;
                }
                evals += (uint64_t)((uint32_t)(w.k - k) - w.multis) + (uint64_t)w.multis * (uint64_t)con->cs;
                evals2 += __reduce_add_sync(FULL, (lane & 7) == 0 ? w.two_l : 0u);
                k = w.k;
                round_k = k;
            }
            if (lane == 0) {
                ctl->k = k;
                ctl->count = stop ? 0 : min(k_end - k, KT);
            }
        }
        __syncthreads();
        if (ctl->count == 0) break;
    }
    if (warp == 0 && owner) store_replica<WPL, 32>(a, E, k, evals, evals2, lane);
    // the other CTAs' copies stay in their shared memory until every CTA
    // of the cluster has made its last remote write into this one
    if constexpr (CL > 1) cg::this_cluster().sync();
}

// Register budget per thread; it sets how many replica warps an SM holds.
// An SM's registers are split between its four schedulers (16384 each): 80
// registers per thread give 6 warps per scheduler, 96 give 5, 112 and 128
// give 4.  The one-row kernels take the smallest budget without spills:
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
#ifndef XW_ANNEAL_MAXNREG_HYBRID
#define XW_ANNEAL_MAXNREG_HYBRID 168
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

// The hybrid form of the large-order kernel (orders up to 448, W in shared
// memory, G in HBM): the same loop.
template <bool GEN>
__global__ void __maxnreg__(XW_ANNEAL_MAXNREG_HYBRID) anneal_hybrid_kernel(AnnealArgs a) {
    for (uint32_t e = threadIdx.x; e < 256; e += blockDim.x) {
        reinterpret_cast<uint2*>(xw_smem)[e] = nibble_entry(e);
        reinterpret_cast<uint32_t*>(xw_smem + 2048)[e] = nibble_entry_bytes(e);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint32_t slot = kNibbleTable + (threadIdx.x >> 5) * a.slot_bytes;
    const uint64_t total = (uint64_t)a.n_items * a.chunks;
    for (;;) {
        uint32_t item = 0;
        if (lane == 0) item = atomicAdd(a.counter, 1u);
        item = __shfl_sync(FULL, item, 0);
        if (item >= total) break;
        const uint32_t c = a.chunks == 1 ? 0u : item / a.n_items;
        const uint32_t rid = a.items[item - c * a.n_items];
        const uint64_t lo = a.iters * c / a.chunks, hi = a.iters * (c + 1) / a.chunks;
        RepHeader* H = reinterpret_cast<RepHeader*>(a.arena + a.rec_off[rid]);
        const bool chunked = a.chunks > 1;
        const bool ok = !chunked || chunk_begin(a.chunk_done + rid, c, a.chunk_wait_ns, &H->err, lane, FULL);
        if (ok) run_replica<16, GEN, 32, false>(a, rid, slot, lane, hi - lo);
        if (chunked) chunk_end(a.chunk_done + rid, c, ok, lane, FULL);
    }
}

// The latency mode: one CTA (CL = 1, a persistent loop over the launch's
// replicas) or one cluster of CL CTAs (one replica per cluster) per replica.
template <bool GEN, int CL, bool ONEZ>
__global__ void __launch_bounds__(512, 1) anneal_spec_kernel(AnnealArgs a, int K) {
    __shared__ uint32_t s_item;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    if constexpr (CL > 1) {
        const uint32_t item = blockIdx.x / CL;
        if (item < a.n_items) run_replica_spec<1, GEN, CL, ONEZ>(a, a.items[item], warp, K, lane);
    } else {
        for (;;) {
            if (threadIdx.x == 0) s_item = atomicAdd(a.counter, 1u);
            __syncthreads();
            const uint32_t item = s_item;
            if (item >= a.n_items) break;
            run_replica_spec<1, GEN, 1, ONEZ>(a, a.items[item], warp, K, lane);
            __syncthreads();
        }
    }
}

// One thread per tempering job: adjacent-rung sweep of
// xweigh_anneal.hpp:1187-1221 on the device draw stream.
__global__ void exchange_kernel(XwJob* jobs, int njobs, uint8_t* arena, const uint64_t* rec_off,
                                const double* ladder, int stop_on_solve) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= njobs) return;
    XwJob& J = jobs[j];
    if (!J.tempering || J.done || (stop_on_solve && J.solved) || J.replicas < 2 || J.replicas > XW_MAX_RUNGS) return;
    const int R = J.replicas;
    if (J.exchange_iters) {
        // served jobs run launches shorter than the exchange interval: swap
        // only at the interval's boundaries of the job's own iteration count
        const uint64_t it0 = reinterpret_cast<const RepHeader*>(arena + rec_off[J.rep_begin])->it;
        if (it0 == 0 || it0 % J.exchange_iters) return;
    }
    int owner[XW_MAX_RUNGS];
    int64_t E[XW_MAX_RUNGS];
    for (int k = 0; k < R; ++k) {
        const RepHeader* H = reinterpret_cast<const RepHeader*>(arena + rec_off[J.rep_begin + k]);
        if (H->rung < 0 || H->rung >= R) return;
        owner[H->rung] = k;
        E[k] = H->obj_total;
    }
    const double* lad = ladder + J.ladder_off;
    const uint64_t round = J.exch_round;
    for (int rung = 0; rung + 1 < R; ++rung) {
        const int ra = owner[rung], rb = owner[rung + 1];
        const double x = __dmul_rn(__dsub_rn(__ddiv_rn(1.0, lad[rung]), __ddiv_rn(1.0, lad[rung + 1])),
                                   (double)(E[ra] - E[rb]));
        bool accept = x >= 0.0;
        if (!accept) {
            const uint4 blk = philox4x32_10(
                make_uint4((uint32_t)rung / 4u, (uint32_t)round, (uint32_t)(round >> 32), 0x80000000u),
                J.key0, J.key1);
            accept = __dmul_rn((double)pick(blk, rung % 4), 0x1p-32) < acceptance_exp(x);
        }
        if (accept) {
            owner[rung] = rb;
            owner[rung + 1] = ra;
        }
    }
    for (int rung = 0; rung < R; ++rung) {
        RepHeader* H = reinterpret_cast<RepHeader*>(arena + rec_off[J.rep_begin + owner[rung]]);
        H->rung = rung;
        H->temperature = lad[rung];
    }
    J.exch_round = round + 1;
}

// One warp per job: best replica by (best score, best conflicts, replica
// index) -- select_best_replica, xweigh_cuda.cu:1342-1354 -- summed
// counters, and a copy of the best replica's best W into a compact buffer.
// The first solver -- least (solve iteration, replica index) among replicas
// whose best score is 0 -- does not depend on how long the job ran after
// it; with first_solver_state its best W is the one copied out.
__global__ void collect_kernel(const XwJob* jobs, int njobs, const uint8_t* arena, const uint64_t* rec_off,
                               const uint64_t* best_out_off, JobOut* out, int8_t* best_out,
                               int first_solver_state) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= njobs) return;
    const XwJob& J = jobs[warp];
    int64_t bs = INT64_MAX, bc = INT64_MAX;
    int br = 0x7fffffff;
    uint64_t moves = 0, evals = 0, iters = 0, acc = 0, acc_rows = 0, evals2 = 0;
    uint64_t fs_it = UINT64_MAX, fs_ns = 0;
    int fs = 0x7fffffff;
    uint32_t err = 0;
#pragma unroll 2
    for (int r = lane; r < J.replicas; r += 32) {
        const RepHeader* H = reinterpret_cast<const RepHeader*>(arena + rec_off[J.rep_begin + r]);
        const int64_t s = H->best_score, c = H->best_conflicts;
        if (s < bs || (s == bs && (c < bc || (c == bc && r < br)))) { bs = s; bc = c; br = r; }
        if (s == 0 && (H->solve_it < fs_it || (H->solve_it == fs_it && r < fs))) {
            fs_it = H->solve_it; fs_ns = H->solve_ns; fs = r;
        }
        moves += H->moves;
        evals += H->cand_evals;
        acc += H->accepted;
        acc_rows += H->accepted_rows;
        evals2 += H->two_row_evals;
        iters = iters > H->it ? iters : H->it;
        err |= H->err;
    }
    for (int off = 16; off > 0; off >>= 1) {
        const int64_t s2 = __shfl_xor_sync(FULL, bs, off), c2 = __shfl_xor_sync(FULL, bc, off);
        const int r2 = __shfl_xor_sync(FULL, br, off);
        if (s2 < bs || (s2 == bs && (c2 < bc || (c2 == bc && r2 < br)))) { bs = s2; bc = c2; br = r2; }
        moves += __shfl_xor_sync(FULL, moves, off);
        evals += __shfl_xor_sync(FULL, evals, off);
        acc += __shfl_xor_sync(FULL, acc, off);
        acc_rows += __shfl_xor_sync(FULL, acc_rows, off);
        evals2 += __shfl_xor_sync(FULL, evals2, off);
        const uint64_t i2 = __shfl_xor_sync(FULL, iters, off);
        iters = iters > i2 ? iters : i2;
        err |= __shfl_xor_sync(FULL, err, off);
        const uint64_t fi2 = __shfl_xor_sync(FULL, fs_it, off), fn2 = __shfl_xor_sync(FULL, fs_ns, off);
        const int f2 = __shfl_xor_sync(FULL, fs, off);
        if (fi2 < fs_it || (fi2 == fs_it && f2 < fs)) { fs_it = fi2; fs_ns = fn2; fs = f2; }
    }
    if (first_solver_state && fs < J.replicas) br = fs;
    if (lane == 0) {
        JobOut o;
        o.score = bs; o.conflicts = bc; o.best_replica = br;
        o.solved = J.solved; o.err = (int32_t)err;
        o.first_solver = fs < J.replicas ? fs : -1;
        o.moves = moves; o.cand_evals = evals; o.iters = iters;
        o.accepted = acc; o.accepted_rows = acc_rows; o.two_row_evals = evals2;
        o.solved_it = fs < J.replicas ? fs_it : 0;
        o.solve_ns = fs < J.replicas ? fs_ns : 0;
        out[warp] = o;
    }
    if (best_out && br >= 0 && br < J.replicas) {
        const uint8_t* src = arena + rec_off[J.rep_begin + br] + J.off_best;
        int8_t* dst = best_out + best_out_off[warp];
        const int nn = J.n * J.n;
        int i = 0;
        if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0) {
            const uint4* s16 = reinterpret_cast<const uint4*>(src);
            for (int k = lane; k < nn / 16; k += 128) {
                uint4 v[4];
                for (int e = 0; e < 4; ++e)
                    if (k + 32 * e < nn / 16) v[e] = s16[k + 32 * e];
                for (int e = 0; e < 4; ++e)
                    if (k + 32 * e < nn / 16) reinterpret_cast<uint4*>(dst)[k + 32 * e] = v[e];
            }
            i = nn & ~15;
        }
        for (i += lane; i < nn; i += 32) dst[i] = (int8_t)src[i];
    }
}

__global__ void mark_t0_kernel(uint64_t* t0) {
    if (*t0 == 0) *t0 = globaltimer();
}

__global__ void stamp_kernel(uint64_t* t) { *t = globaltimer(); }

}  // namespace

uint32_t anneal_slot_bytes(int n, int m, int opl) {
    if (opl <= 4) return packed_slot_bytes(n, m, opl);
    // Above order 128 a slot keeps the size that W, a 16-bit Gram matrix with
    // a padded row, 256-bit row masks and the per-warp buffers took, so that
    // the same orders and weights fit the device's shared memory as ever
    const uint32_t N = (uint32_t)n;
    const uint32_t kept = xw_pad16(N * N) + xw_pad16(2u * N * (N | 1u)) + xw_pad16(4u * N) + xw_pad16(N * (uint32_t)m) +
                          32u * N + 1184u;
    return std::max(kept, packed_slot_bytes(n, m, 8));
}

// rows per lane; W(128,128) has off-diagonal Gram entries of +-128, which a
// signed byte does not hold, and takes the 16-bit kernel of the orders above
int anneal_opl(int n, int w) { return n <= 32 ? 1 : n <= 64 ? 2 : n <= 128 && w < 128 ? 4 : 8; }

const void* anneal_kernel_fn(int opl, bool general, int rpw, bool one_zero) {
    if (one_zero && opl == 1 && rpw == 1) {
        return general ? reinterpret_cast<const void*>(&anneal_kernel<1, true, 32, true>)
                       : reinterpret_cast<const void*>(&anneal_kernel<1, false, 32, true>);
    }
    if (rpw == 2) {
        return general ? reinterpret_cast<const void*>(&anneal_kernel<1, true, 16>)
                       : reinterpret_cast<const void*>(&anneal_kernel<1, false, 16>);
    }
    if (general) {
        if (opl == 1) return reinterpret_cast<const void*>(&anneal_kernel<1, true, 32>);
        if (opl == 2) return reinterpret_cast<const void*>(&anneal_kernel<2, true, 32>);
        if (opl == 4) return reinterpret_cast<const void*>(&anneal_kernel<4, true, 32>);
        return reinterpret_cast<const void*>(&anneal_kernel<8, true, 32>);
    }
    if (opl == 1) return reinterpret_cast<const void*>(&anneal_kernel<1, false, 32>);
    if (opl == 2) return reinterpret_cast<const void*>(&anneal_kernel<2, false, 32>);
    if (opl == 4) return reinterpret_cast<const void*>(&anneal_kernel<4, false, 32>);
    return reinterpret_cast<const void*>(&anneal_kernel<8, false, 32>);
}

uint32_t anneal_hybrid_slot_bytes(int n, int m) { return hybrid_slot_bytes(n, m); }

uint64_t anneal_hybrid_arena_bytes(int n) { return hybrid_arena(n).bytes; }

uint32_t anneal_hybrid_table_bytes() { return kNibbleTable; }

const void* anneal_hybrid_kernel_fn(bool general) {
    return general ? reinterpret_cast<const void*>(&anneal_hybrid_kernel<true>)
                   : reinterpret_cast<const void*>(&anneal_hybrid_kernel<false>);
}

cudaError_t launch_anneal(const AnnealArgs& args, int opl, bool general, int warps_per_block, int blocks,
                          cudaStream_t stream, int rpw) {
    if (rpw != 1 && (rpw != 2 || opl != 1)) return cudaErrorInvalidValue;
    const size_t smem = (size_t)warps_per_block * rpw * args.slot_bytes;
    const dim3 grid(blocks), block(32 * warps_per_block);
    void* kargs[] = {const_cast<AnnealArgs*>(&args)};
    return cudaLaunchKernel(anneal_kernel_fn(opl, general, rpw, args.one_zero != 0), grid, block,
                            kargs, smem, stream);
}

// wpr warps per replica on `ctas` CTAs (1, 2 or 4; a cluster above 1) of
// wpr / ctas warps each
uint32_t anneal_spec_cta_bytes(uint32_t slot_bytes, int wpr, int ctas) {
    return spec_layout(slot_bytes, wpr / ctas, ctas).bytes;
}

template <bool ONEZ>
const void* spec_fn(bool general, int ctas) {
    if (ctas == 4)
        return general ? reinterpret_cast<const void*>(&anneal_spec_kernel<true, 4, ONEZ>)
                       : reinterpret_cast<const void*>(&anneal_spec_kernel<false, 4, ONEZ>);
    if (ctas == 2)
        return general ? reinterpret_cast<const void*>(&anneal_spec_kernel<true, 2, ONEZ>)
                       : reinterpret_cast<const void*>(&anneal_spec_kernel<false, 2, ONEZ>);
    return general ? reinterpret_cast<const void*>(&anneal_spec_kernel<true, 1, ONEZ>)
                   : reinterpret_cast<const void*>(&anneal_spec_kernel<false, 1, ONEZ>);
}

const void* anneal_spec_kernel_fn(bool general, int ctas, bool one_zero) {
    return one_zero ? spec_fn<true>(general, ctas) : spec_fn<false>(general, ctas);
}

cudaError_t launch_anneal_spec(const AnnealArgs& args, bool general, int wpr, int ctas, int blocks,
                               cudaStream_t stream) {
    const int CL = ctas;
    if ((CL != 1 && CL != 2 && CL != 4) || wpr % CL != 0 || wpr / CL < 2 || wpr / CL > 16 || args.chunks != 1)
        return cudaErrorInvalidValue;
    int k = wpr / CL;
    void* kargs[] = {const_cast<AnnealArgs*>(&args), &k};
    if (CL == 1)
        return cudaLaunchKernel(anneal_spec_kernel_fn(general, 1, args.one_zero != 0), dim3(blocks), dim3(32 * k), kargs,
                                args.slot_bytes, stream);
    // one cluster of CL CTAs per replica
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CL * args.n_items);
    cfg.blockDim = dim3(32 * k);
    cfg.dynamicSmemBytes = args.slot_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, anneal_spec_kernel_fn(general, CL, args.one_zero != 0), kargs);
}

cudaError_t launch_exchange(XwJob* jobs, int njobs, uint8_t* arena, const uint64_t* rec_off, const double* ladder,
                            int stop_on_solve, cudaStream_t stream) {
    if (njobs <= 0) return cudaSuccess;
    exchange_kernel<<<(njobs + 127) / 128, 128, 0, stream>>>(jobs, njobs, arena, rec_off, ladder, stop_on_solve);
    return cudaGetLastError();
}

cudaError_t launch_collect(const XwJob* jobs, int njobs, const uint8_t* arena, const uint64_t* rec_off,
                           const uint64_t* best_out_off, JobOut* out, int8_t* best_out, cudaStream_t stream,
                           int first_solver_state) {
    if (njobs <= 0) return cudaSuccess;
    collect_kernel<<<(njobs + 3) / 4, 128, 0, stream>>>(jobs, njobs, arena, rec_off, best_out_off, out, best_out,
                                                        first_solver_state);
    return cudaGetLastError();
}

cudaError_t launch_stamp(uint64_t* t, cudaStream_t stream) {
    stamp_kernel<<<1, 1, 0, stream>>>(t);
    return cudaGetLastError();
}

cudaError_t launch_mark_t0(uint64_t* t0, cudaStream_t stream) {
    mark_t0_kernel<<<1, 1, 0, stream>>>(t0);
    return cudaGetLastError();
}

}  // namespace xw
