// One training step of the learned AO's network on host arrays, in a build of any feature step count.
#include "../megamol_gb300/csrc/mlp_internal.h"

using namespace p2v;

extern "C" __attribute__((visibility("default"))) int inputs() {
    return MLP_IN;
}

// grad: MLP_NPARAM + 1 floats (the summed loss last)
extern "C" __attribute__((visibility("default"))) int train_step(const float* P, const float* X, const float* T, int n,
                                                                 float* grad) {
    const int blocks = mlp_train_blocks(n);
    const size_t size[6] = {MLP_NPARAM, (size_t) n * MLP_IN, (size_t) n, (size_t) blocks * MLP_NPARAM, (size_t) blocks,
                            MLP_NPARAM + 1};
    float* d[6] = {};
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < 6 && e == cudaSuccess; ++k) {
        e = cudaMalloc(&d[k], sizeof(float) * size[k]);
        if (e == cudaSuccess)
            e = cudaMemset(d[k], 0xFF, sizeof(float) * size[k]);  // NaN: whatever is not written shows
    }
    const float* src[3] = {P, X, T};
    for (int k = 0; k < 3 && e == cudaSuccess; ++k)
        e = cudaMemcpy(d[k], src[k], sizeof(float) * size[k], cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = launch_mlp_train_step(d[0], d[1], d[2], nullptr, n, d[3], d[4], d[5], nullptr);
    if (e == cudaSuccess)
        e = cudaMemcpy(grad, d[5], sizeof(float) * size[5], cudaMemcpyDeviceToHost);
    for (float* p : d)
        cudaFree(p);
    return (int) e;
}
