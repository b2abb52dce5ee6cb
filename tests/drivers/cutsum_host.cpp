// The exact float sums of mdsm_gb300/csrc/cutsum.cuh on the host, in the batches that the clip's
// statistics feed them: whole 32s as two batches of 16, then single samples.
#include "cuda_runtime.h"

#include "cutsum.cuh"

extern "C" int cut_sum(const float *x, int n, float biggest, double *sum)
{
    mdsm::CutSum cs;
    cs.start(biggest);
    int i = 0;
    for (; i + 32 <= n; i += 32)
        for (int h = 0; h < 2; ++h) {
            float v[16];
            memcpy(v, x + i + 16 * h, sizeof v);
            cs.add(v);
        }
    for (; i < n; ++i) {
        const float v[1] = {x[i]};
        cs.add(v);
    }
    *sum = cs.sum();
    return cs.ok();
}
