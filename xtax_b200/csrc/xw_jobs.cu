// xw_jobs.cu -- the kernels over whole jobs beside the annealing kernels:
// tempering exchanges, collecting results, time stamps.  A module of its own,
// small, since every batch uses it.
#include <cuda_runtime.h>

#include "xw_device.cuh"
#include "xw_kernels.h"

namespace xw {

namespace {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ uint64_t globaltimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
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
