// xw_anneal.cu -- the population annealing kernel for weighing matrices: its
// instantiations for orders up to 32, and its launches.
//
// One warp (or a half-warp) owns one replica at a time, its state in the
// warp's shared-memory slot; the whole iteration is warp-synchronous: no
// __syncthreads, no block-wide reductions.  The replica loop is in
// xw_replica.cuh, the iteration itself in xw_packed.cuh: rows of W and G
// packed into words, bytes of G up to order 128, halfwords above.
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
#include <algorithm>

#include "xw_replica.cuh"

namespace xw {

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
    if (opl != 1) return anneal_wide_kernel_fn(opl, general);
    return general ? reinterpret_cast<const void*>(&anneal_kernel<1, true, 32>)
                   : reinterpret_cast<const void*>(&anneal_kernel<1, false, 32>);
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

}  // namespace xw
