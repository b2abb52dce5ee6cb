// Which kernel a brute-force stage launches with and without the rows' moments, on the host: the launch is
// recorded instead of made.  Arguments: type, channels, samples, trials, step (pc cm^-3).  Prints
// "sums <a> moments <b>", a and b each gs (group sums) or packed.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "internal.h"

static size_t g_smem;

extern "C" cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t smem, cudaStream_t)
{
    g_smem = smem;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
extern "C" cudaError_t cudaMemset2DAsync(void *, size_t, int, size_t, size_t, cudaStream_t)
{
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError(void) { return cudaSuccess; }

int main(int, char **argv)
{
    mdsm::StageGeom g;
    g.in_dtype = std::atoi(argv[1]);
    g.nchans = std::atoi(argv[2]);
    g.nsamp = std::atoi(argv[3]);
    g.ndms = std::atoi(argv[4]);
    g.ngroups = 1;
    g.acc_int = g.out_i32 = 1;
    g.DPW = 4;
    std::vector<int32_t> S((size_t)g.ndms * g.nchans);
    for (int d = 0; d < g.ndms; ++d)
        for (int c = 0; c < g.nchans; ++c) {
            const double f = 1500.0 - 300.0 / g.nchans * c;
            S[(size_t)d * g.nchans + c] = (int32_t)std::floor(
                4148.741601 * (1.0 / (f * f) - 1.0 / (1500.0 * 1500.0)) * std::atof(argv[5]) * d / 64e-6);
        }
    if (mdsm::build_stage_tables(g, S) != MDSM_OK || mdsm::gs_build(g, S) != MDSM_OK) return 1;
    unsigned long long mom;
    for (int k = 0; k < 2; ++k) {
        g_smem = 0;
        if (mdsm::launch_stage(g, nullptr, 1 << 20, 0, nullptr, 1 << 20, 0, nullptr, nullptr, nullptr, -1,
                               k ? &mom : nullptr, g.ndms) != MDSM_OK)
            return 1;
        const bool gs = g.gs.shape >= 0 && g_smem == g.gs.smem;
        if (!gs && g_smem != g.smem_bytes) return 1;
        std::printf("%s %s ", k ? "moments" : "sums", gs ? "gs" : "packed");
    }
    std::printf("\n");
    return 0;
}
