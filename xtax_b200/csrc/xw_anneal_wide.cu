// xw_anneal_wide.cu -- the annealing kernels of orders above 32: two, four and
// eight rows a lane (xw_replica.cuh), and the hybrid form of the large orders
// (257..448: W in shared memory, G in HBM).
#include "xw_replica.cuh"

namespace xw {

namespace {

#ifndef XW_ANNEAL_MAXNREG_HYBRID
#define XW_ANNEAL_MAXNREG_HYBRID 168
#endif
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

}  // namespace

const void* anneal_wide_kernel_fn(int opl, bool general) {
    if (general) {
        if (opl == 2) return reinterpret_cast<const void*>(&anneal_kernel<2, true, 32>);
        if (opl == 4) return reinterpret_cast<const void*>(&anneal_kernel<4, true, 32>);
        return reinterpret_cast<const void*>(&anneal_kernel<8, true, 32>);
    }
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

}  // namespace xw
