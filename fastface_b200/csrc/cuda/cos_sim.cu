// cos_sim.cu -- cosine-similarity matrix of two sets of 512-d embeddings.
//
// out[i][j] = CosSim(a[i], b[j]) with the arithmetic of the reference's Go wrapper
// (go/fastface/fastface.go:157-168): dot product and both squared norms accumulated in
// float64 in index order, 0 when a norm is 0, result rounded to float32 once at the end.  A
// float32 x float32 product is exact in float64 (48 bits), so one fused multiply-add per step rounds exactly where
// "dot += x * y" does: the kernel reproduces the host function bit for bit.
//
// Bound: float64 FMA (64 per cycle and SM) from a few hundred rows up, copies below and around it.  A block of 256
// threads computes 16 * RM x 64 outputs, RM x 4 per thread, from operands converted to float64 once per block and
// staged CS_KC dimensions at a time; its first threads carry the norms of the block's rows along (one FMA per
// dimension each), so every norm is computed once per block and not once per pair.
// 1024 x 1024 from and to pageable host arrays: 3060 -> 620 us a call (three allocations and frees a call, norms summed
// per pair and separate multiplies and adds before); what is left is the copies.
#include "ffcu_internal.cuh"
#include "cos_sim.cuh"

#include <algorithm>
#include <new>

#define CS_DIM 512
#define CS_KC 16
#define CS_TJ 64

// Rows of a tile lie CS_PAD doubles apart per dimension: [k][row], so a thread's 4 rows are 32 contiguous bytes.
template <int RM>
__global__ void __launch_bounds__(256) cos_sim_matrix_kernel(const float* __restrict__ a, int n, const float* __restrict__ b, int m,
                                                             float* __restrict__ out, size_t pitch)
{
    constexpr int TI = 16 * RM;
    __shared__ alignas(16) double sa[CS_KC][TI + 2], sb[CS_KC][CS_TJ + 2];
    __shared__ double na[TI], nb[CS_TJ];                   // square roots of the squared norms
    const int t = threadIdx.x, tx = t % 16, ty = t / 16;
    const int i0 = blockIdx.y * TI, j0 = blockIdx.x * CS_TJ;
    double acc[RM][4] = {};
    double nrm = 0.0;
    for (int k0 = 0; k0 < CS_DIM; k0 += CS_KC) {
        for (int e = t; e < (TI + CS_TJ) * (CS_KC / 4); e += 256) {
            const int r = e / (CS_KC / 4), c = e % (CS_KC / 4) * 4;
            const bool is_a = r < TI;
            const int row = is_a ? i0 + r : j0 + r - TI;
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (row < (is_a ? n : m)) v = __ldg((const float4*)((is_a ? a : b) + (size_t)row * CS_DIM + k0 + c));
            double* d = is_a ? &sa[c][r] : &sb[c][r - TI];
            const int ld = is_a ? TI + 2 : CS_TJ + 2;
            d[0] = (double)v.x; d[ld] = (double)v.y; d[2 * ld] = (double)v.z; d[3 * ld] = (double)v.w;
        }
        __syncthreads();
        if (t < TI + CS_TJ) {
            const double* p = t < TI ? &sa[0][t] : &sb[0][t - TI];
            const int ld = t < TI ? TI + 2 : CS_TJ + 2;
#pragma unroll
            for (int k = 0; k < CS_KC; k++) nrm = __fma_rn(p[k * ld], p[k * ld], nrm);
        }
#pragma unroll
        for (int k = 0; k < CS_KC; k++) {
            double x[RM], y[4];
#pragma unroll
            for (int r = 0; r < RM; r++) x[r] = sa[k][ty * RM + r];
#pragma unroll
            for (int c = 0; c < 4; c++) y[c] = sb[k][tx * 4 + c];
#pragma unroll
            for (int r = 0; r < RM; r++)
#pragma unroll
                for (int c = 0; c < 4; c++) acc[r][c] = __fma_rn(x[r], y[c], acc[r][c]);
        }
        __syncthreads();
    }
    if (t < TI + CS_TJ) (t < TI ? na[t] : nb[t - TI]) = __dsqrt_rn(nrm);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RM; r++) {
        const int i = i0 + ty * RM + r;
        const double ra = na[ty * RM + r];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int j = j0 + tx * 4 + c;
            const double rb = nb[tx * 4 + c];
            // the square root of a squared norm is 0 exactly where the squared norm is
            const float v = (ra != 0.0 && rb != 0.0) ? (float)__ddiv_rn(acc[r][c], __dmul_rn(ra, rb)) : 0.0f;
            if (i < n && j < m) out[(size_t)i * pitch + j] = v;
        }
    }
}

static void launch_matrix(const float* a, int n, const float* b, int m, float* out, size_t pitch, cudaStream_t s)
{
    // Rows per block: 64 when that fills half the SMs' worth of blocks, else 16 (a handful of queries against a gallery
    // would spend the FMAs on rows that are not there).
    const int gx = (m + CS_TJ - 1) / CS_TJ;
    if (n > 32 && gx * ((n + 63) / 64) >= 74) cos_sim_matrix_kernel<4><<<dim3(gx, (n + 63) / 64), 256, 0, s>>>(a, n, b, m, out, pitch);
    else cos_sim_matrix_kernel<1><<<dim3(gx, (n + 15) / 16), 256, 0, s>>>(a, n, b, m, out, pitch);
}

// One call works in slices of at most CS_MAX_N x CS_MAX_M pairs, so the workspace a context keeps is bounded
// (4 + 8 + 32 MB) whatever the matrix.
#define CS_MAX_N 2048
#define CS_MAX_M 4096

void CosWorkspace::release()
{
    cudaFree(a); cudaFree(b); cudaFree(out);
    if (stream) cudaStreamDestroy(stream);
    a = b = out = nullptr; cap_a = cap_b = cap_out = 0; stream = nullptr;
}

static bool grow(float** p, size_t* cap, size_t need)
{
    if (need <= *cap) return true;
    cudaFree(*p);
    *p = nullptr; *cap = 0;
    if (cudaMalloc(p, need * sizeof(float)) != cudaSuccess) return false;
    *cap = need;
    return true;
}

int CosWorkspace::run(const float* ha, int n, const float* hb, int m, float* hout)
{
    const int sn = std::min(n, CS_MAX_N), sm = std::min(m, CS_MAX_M);
    if ((!stream && cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking) != cudaSuccess) ||
        !grow(&a, &cap_a, (size_t)sn * CS_DIM) || !grow(&b, &cap_b, (size_t)sm * CS_DIM) || !grow(&out, &cap_out, (size_t)sn * sm)) {
        ffcu_set_error("ffcu_cos_sim_matrix: device allocation failed");
        cudaGetLastError();
        return -2;
    }
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < n && e == cudaSuccess; i += sn) {
        const int cn = std::min(sn, n - i);
        e = cudaMemcpyAsync(a, ha + (size_t)i * CS_DIM, (size_t)cn * CS_DIM * 4, cudaMemcpyHostToDevice, stream);
        for (int j = 0; j < m && e == cudaSuccess; j += sm) {
            const int cm = std::min(sm, m - j);
            e = cudaMemcpyAsync(b, hb + (size_t)j * CS_DIM, (size_t)cm * CS_DIM * 4, cudaMemcpyHostToDevice, stream);
            if (e != cudaSuccess) break;
            launch_matrix(a, cn, b, cm, out, (size_t)cm, stream);
            e = cudaGetLastError();
            if (e == cudaSuccess)
                e = cm == m ? cudaMemcpyAsync(hout + (size_t)i * m, out, (size_t)cn * m * 4, cudaMemcpyDeviceToHost, stream)
                            : cudaMemcpy2DAsync(hout + (size_t)i * m + j, (size_t)m * 4, out, (size_t)cm * 4, (size_t)cm * 4, cn,
                                                cudaMemcpyDeviceToHost, stream);
        }
    }
    const cudaError_t e2 = cudaStreamSynchronize(stream);
    if (e == cudaSuccess) e = e2;
    if (e != cudaSuccess) { ffcu_set_error("ffcu_cos_sim_matrix: %s", cudaGetErrorString(e)); return -100; }
    return 0;
}

// a: host [n][512], b: host [m][512], out: host [n][m].  Returns 0 or a negative code.
extern "C" int ffcu_cos_sim_matrix(int device, const float* a, int n, const float* b, int m, float* out)
{
    if (!a || !b || !out || n < 1 || m < 1) { ffcu_set_error("ffcu_cos_sim_matrix: bad arguments"); return -1; }
    FFCU_CHECK(cudaSetDevice(device));
    CosWorkspace w;
    const int rc = w.run(a, n, b, m, out);
    w.release();
    return rc;
}

// The same through a workspace that its owner keeps.  Calls from several threads each go through: one takes the
// workspace, the others make their own for the call.
int CosWorkspace::call(int device, const float* ha, int n, const float* hb, int m, float* hout)
{
    if (!ha || !hb || !hout || n < 1 || m < 1) { ffcu_set_error("ffcu_cos_sim_matrix: bad arguments"); return -1; }
    if (!mu.try_lock()) return ffcu_cos_sim_matrix(device, ha, n, hb, m, hout);
    int rc = cudaSetDevice(device) == cudaSuccess ? 0 : -100;
    if (rc) { ffcu_set_error("cudaSetDevice(%d) failed", device); cudaGetLastError(); }
    else rc = run(ha, n, hb, m, hout);
    mu.unlock();
    return rc;
}
