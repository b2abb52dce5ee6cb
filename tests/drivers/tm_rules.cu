// Whether a plan's float stage takes the tensor-memory kernel, where the runtime reports `argv[1]` registers
// a thread for it (0: it reports an error): prints the chosen shape, -1 for none, and its shared memory.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>

static int g_regs;

static cudaError_t reported_attributes(cudaFuncAttributes *at, const void *)
{
    if (g_regs == 0) return cudaErrorInvalidDeviceFunction;
    *at = cudaFuncAttributes();
    at->numRegs = g_regs;
    return cudaSuccess;
}

#define cudaFuncGetAttributes reported_attributes
#include "tmsum.cu"

int main(int argc, char **argv)
{
    g_regs = argc > 1 ? std::atoi(argv[1]) : 0;
    mdsm::StageGeom g;
    g.nchans = 128;
    g.ndms = argc > 2 ? std::atoi(argv[2]) : 496;
    g.ngroups = 1;
    g.nsamp = argc > 3 ? std::atoi(argv[3]) : 32000;
    g.in_dtype = MDSM_F32;
    g.acc_int = 0;
    g.DPW = 4;
    std::vector<int32_t> S((size_t)g.ndms * g.nchans);
    for (int d = 0; d < g.ndms; ++d)
        for (int c = 0; c < g.nchans; ++c) S[(size_t)d * g.nchans + c] = d * c / 512;
    if (mdsm::build_stage_tables(g, S) != MDSM_OK || mdsm::tm_build(g, S) != MDSM_OK) return 1;
    std::printf("%d %zu\n", g.tm.shape, g.tm.smem);
    return 0;
}
