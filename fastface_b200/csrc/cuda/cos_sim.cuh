// cos_sim.cuh -- device workspace of the similarity matrix (cos_sim.cu): a context keeps one between calls.
#pragma once
#include <cuda_runtime.h>
#include <mutex>

struct CosWorkspace {
    std::mutex mu;                       // held by the call that uses the buffers
    float *a = nullptr, *b = nullptr, *out = nullptr;
    size_t cap_a = 0, cap_b = 0, cap_out = 0;        // floats
    cudaStream_t stream = nullptr;
    int call(int device, const float* ha, int n, const float* hb, int m, float* hout);
    int run(int device, const float* ha, int n, const float* hb, int m, float* hout);
    void release();
};
