// xw_spec_lean.cu -- the latency mode's lean kernels, and its launches.
#include "xw_spec.cuh"

namespace xw {

// wpr warps per replica on `ctas` CTAs (1, 2 or 4; a cluster above 1) of
// wpr / ctas warps each
uint32_t anneal_spec_cta_bytes(uint32_t slot_bytes, int wpr, int ctas) {
    return spec_layout(slot_bytes, wpr / ctas, ctas).bytes;
}

const void* anneal_spec_lean_fn(int ctas, bool one_zero) { return spec_fn<false>(ctas, one_zero); }

const void* anneal_spec_kernel_fn(bool general, int ctas, bool one_zero) {
    return general ? anneal_spec_general_fn(ctas, one_zero) : anneal_spec_lean_fn(ctas, one_zero);
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

}  // namespace xw
