// xw_spec.cuh -- the latency mode: one replica on several warps that speculate
// its next iterations (orders up to 32).  xw_spec_lean.cu and
// xw_spec_general.cu instantiate it, each a module of its own.
#pragma once

#include <cooperative_groups.h>

#include "xw_replica.cuh"

namespace xw {

namespace {

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
// So warp 0 watches the advance: while a round advances by less than it costs
// in steps of the one-warp loop (cost10 below, tenths of a step, measured on
// W(12,11): 2.6 on a cluster, 1.2 + K / 20 on one CTA) it goes on alone, step
// by step, until accepts are rare enough again (in a cluster every CTA's warp 0
// makes the same steps on its copy).

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
        make_env<WPL, GEN, 32, ONEZ>(E, J, 0u, L.off_extra + (uint32_t)(warp - 1) * 512u, lane, GEN ? H->obj_kind : 0);

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
            // of them reaches a cooling or reheat step before the span's last
            // call, so when none can, they are counted in bulk and only the
            // accepted move is committed.  Otherwise the ordered walk.
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
            // (a step due at the span's last call, as the launch's end often
            // is, comes after it)
            bool fast = jend <= k_evt - k;
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

// The latency mode's kernel on `ctas` CTAs a replica.
template <bool GEN>
const void* spec_fn(int ctas, bool one_zero) {
    if (ctas == 4)
        return one_zero ? reinterpret_cast<const void*>(&anneal_spec_kernel<GEN, 4, true>)
                        : reinterpret_cast<const void*>(&anneal_spec_kernel<GEN, 4, false>);
    if (ctas == 2)
        return one_zero ? reinterpret_cast<const void*>(&anneal_spec_kernel<GEN, 2, true>)
                        : reinterpret_cast<const void*>(&anneal_spec_kernel<GEN, 2, false>);
    return one_zero ? reinterpret_cast<const void*>(&anneal_spec_kernel<GEN, 1, true>)
                    : reinterpret_cast<const void*>(&anneal_spec_kernel<GEN, 1, false>);
}

}  // namespace

}  // namespace xw
