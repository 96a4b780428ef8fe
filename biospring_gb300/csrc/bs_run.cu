// bs_run.cu -- launch of the kernels of several steps (bs_run.cuh).

#include "bs_kernels.cuh"

namespace bsg
{

static const void *run_kernel(const Params &p)
{
    const bool lean = lean_step(p);
    const int hold = p.run_hold;
    switch (p.steric_mode)
    {
    case BS_STERIC_LINEAR:
        return run_linear(p.step_lanes, lean, hold);
    case BS_STERIC_LJ_12_6_AMBER:
        return run_amber(p.step_lanes, lean, hold);
    case BS_STERIC_LJ_8_6_LEWITT:
        return run_lewitt(p.step_lanes, lean, hold);
    case BS_STERIC_LJ_8_6_ZACHARIAS:
        return run_zacharias(p.step_lanes, lean, hold);
    default:
        return nullptr;
    }
}

int run_blocks(const Params &p)
{
    return static_cast<int>((static_cast<long long>(p.n) * p.step_lanes + kStepKernelBlock - 1) / kStepKernelBlock);
}

cudaError_t run_fits(Params &p)
{
    p.run_on = p.run_hold = 0;
    int dev = 0, sms = 0, coop = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    // the form with the most registers that is resident at once
    const int forms[3] = {2, 3, 0};
    for (int f = 0; f < 3 && !p.run_on && e == cudaSuccess && coop && p.nsys == 0; ++f)
    {
        p.run_hold = forms[f];
        const void *fn = run_kernel(p);
        if (!fn)
            continue;
        int per_sm = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kStepKernelBlock, 0);
        p.run_on = e == cudaSuccess && run_blocks(p) <= per_sm * sms;
    }
    return e;
}

cudaError_t launch_run(const Params &p, int count, cudaStream_t st, float4 *save, float4 *save_lo)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(run_blocks(p)));
    cfg.blockDim = dim3(kStepKernelBlock);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void *args[] = {const_cast<Params *>(&p), &count, &save, &save_lo};
    return cudaLaunchKernelExC(&cfg, run_kernel(p), args);
}

} // namespace bsg
