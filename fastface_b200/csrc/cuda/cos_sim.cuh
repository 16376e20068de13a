// cos_sim.cuh -- workspace of the similarity matrix (cos_sim.cu): a context keeps one between calls.
#pragma once
#include <cuda_runtime.h>
#include <mutex>

struct ff_copy_pool;

#define CS_PIECES 4                      // page-locked ring either way, pieces of CS_PIECE bytes
#define CS_PIECE ((size_t)1 << 20)

struct CosWorkspace {
    std::mutex mu;                       // held by the call that uses the buffers
    float *a = nullptr, *b = nullptr, *out = nullptr;
    size_t cap_a = 0, cap_b = 0, cap_out = 0;        // floats
    cudaStream_t stream = nullptr;
    // What a kept workspace has besides: made by its first call, page-locked memory as far as the host gives it
    bool tried = false;
    char *pin_in = nullptr, *pin_out = nullptr;
    ff_copy_pool* pool = nullptr;
    cudaStream_t s_in = nullptr, s_out = nullptr;
    cudaEvent_t ev_in[CS_PIECES] = {}, ev_out[CS_PIECES] = {}, ev_uploaded = nullptr, ev_done[2] = {};
    unsigned pieces_in = 0;
    int call(int device, const float* ha, int n, const float* hb, int m, float* hout);
    int run(int device, const float* ha, int n, const float* hb, int m, float* hout);
    void release();
private:
    bool pipeline_ready();
    int run_pipeline(int n_sm, const float* ha, int n, const float* hb, int m, float* hout, bool in_a, bool in_b, bool out_staged);
    cudaError_t upload(float* dst, const float* src, size_t bytes, bool staged);
    cudaError_t deliver(float* hout, size_t pitch, const float* src, int rows, int cols, bool staged, cudaEvent_t done);
};
