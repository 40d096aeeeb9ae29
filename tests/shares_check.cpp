// bc1_shares.h's rules as plain functions (built and called by tests/test_shares.py).
#include "../icbc_gb300/csrc/bc1_shares.h"

extern "C" {
void batch(const int *levels, const int64_t *blocks, int n, int64_t warps, int level_kernels, int *sizes, int *ctas) {
    const icbc_gpu::BatchShape s = icbc_gpu::batch_shape(levels, blocks, n, warps, level_kernels != 0);
    for (int l = 0; l < 10; l++) sizes[l] = s.task_blocks[l], ctas[l] = s.cta_warps[l];
}
int bands(int level, int64_t blocks, int sms) { return icbc_gpu::host_bands(level, blocks, sms); }
int image(int64_t n, int64_t workers, int level) { return icbc_gpu::image_share(n, workers, level); }
}
