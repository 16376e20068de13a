// cos_sim.cu -- cosine-similarity matrix of two sets of 512-d embeddings.
//
// out[i][j] = CosSim(a[i], b[j]) with the arithmetic of the reference's Go wrapper
// (go/fastface/fastface.go:157-168): dot product and both squared norms accumulated in
// float64 in index order, 0 when a norm is 0, result rounded to float32 once at the end.  A
// float32 x float32 product is exact in float64 (48 bits), so one fused multiply-add per step rounds exactly where
// "dot += x * y" does: the kernel reproduces the host function bit for bit.
//
// Bound: latency.  A pair's sum is a chain of 512 dependent float64 FMAs, with its shared-memory reads about 10 us however
// small the matrix; with many blocks the shared-memory data path is two thirds busy and the float64 pipe 44 % (64 x 64 outputs a
// block, 1024 x 1000).  Everything else is arranged around that chain: the operands of the next CS_KC
// dimensions are fetched into registers while the current ones are used, converted to float64 once per block and stored into the
// other of two shared buffers (one barrier per chunk), and the norms have warps of their own, one row a thread, so that
// their chains run beside the pairs'.  Rows lie KC + 2 doubles apart: 16-byte reads of two dimensions at eight
// consecutive rows touch every bank once, and a warp's 4 x 8 lanes read 4 rows of `a` and 8 of `b` for each 32 sums.
//
// Kernel times, us, one output a thread and no prefetch | 16 x 64 or 64 x 64 outputs a block, norms in front of each chunk's
// sums | this kernel: 1 x 100 24.7 | 61.6 | 12.5, 24 x 300 26.8 | 61.6 | 12.4, 64 x 1000 32.9 | 61.6 | 20.7, 1 x 10000 59 | 98 | 45,
// 128 x 1000 51.4 | 61.6 | 22.6, 256 x 1000 82 | 72 | 37, 1024 x 1000 287 | 119 | 95, 1024 x 10000 2656 | 884 | 779.  Calls (pageable arrays, copies included): 1 x 100 90 | 115 | 57,
// 16 x 300 120 | 137 | 78, 128 x 300 146 | 156 | 108, 256 x 1000 1613 | 359 | 295, 1024 x 1000 2643 | 643 | 617.
#include "ffcu_internal.cuh"
#include "cos_sim.cuh"

#include <stdint.h>
#include <algorithm>

#define CS_DIM 512

// WR x WC warps of 4 x 8 lanes, RM x RN pairs per thread (rows 4 apart, columns 8 apart), KC dimensions at a time.
template <int WR, int WC, int RM, int RN, int KC>
struct CosTile {
    static constexpr int TI = WR * 4 * RM, TJ = WC * 8 * RN, ROWS = TI + TJ;
    static constexpr int PAIR_THREADS = 32 * WR * WC;
    static constexpr int THREADS = PAIR_THREADS + (ROWS + 31) / 32 * 32;       // then one thread per row for the norms
    static constexpr int VECS = KC / 4, FETCH = (ROWS * VECS + THREADS - 1) / THREADS;
};

template <int WR, int WC, int RM, int RN, int KC>
__global__ void __launch_bounds__(CosTile<WR, WC, RM, RN, KC>::THREADS)
cos_sim_matrix_kernel(const float* __restrict__ a, int n, const float* __restrict__ b, int m, float* __restrict__ out, size_t pitch)
{
    using T = CosTile<WR, WC, RM, RN, KC>;
    __shared__ alignas(16) double s[2][T::ROWS][KC + 2];   // rows of a, then rows of b
    __shared__ double root[T::ROWS];                       // square roots of the squared norms
    const int t = threadIdx.x, warp = t / 32, lane = t % 32;
    const int i0 = blockIdx.y * T::TI, j0 = blockIdx.x * T::TJ;
    float4 v[T::FETCH];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int u = 0; u < T::FETCH; u++) {
            const int e = t + u * T::THREADS, r = e / T::VECS, c = e % T::VECS * 4;
            v[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (r < T::ROWS) {
                const bool is_a = r < T::TI;
                const int row = is_a ? i0 + r : j0 + r - T::TI;
                if (row < (is_a ? n : m)) v[u] = __ldg((const float4*)((is_a ? a : b) + (size_t)row * CS_DIM + k0 + c));
            }
        }
    };
    auto put = [&](int buf) {
#pragma unroll
        for (int u = 0; u < T::FETCH; u++) {
            const int e = t + u * T::THREADS, r = e / T::VECS, c = e % T::VECS * 4;
            if (r < T::ROWS) {
                double2* d = (double2*)&s[buf][r][c];
                d[0] = make_double2((double)v[u].x, (double)v[u].y);
                d[1] = make_double2((double)v[u].z, (double)v[u].w);
            }
        }
    };
    const int ri = warp / WC * 4 * RM + lane / 8, cj = warp % WC * 8 * RN + lane % 8;      // of this thread's first pair
    const int norm_row = t - T::PAIR_THREADS;
    double acc[RM][RN] = {};
    double nrm = 0.0;
    fetch(0);
    put(0);
    for (int k0 = 0; k0 < CS_DIM; k0 += KC) {
        const int buf = k0 / KC & 1;
        const bool more = k0 + KC < CS_DIM;
        __syncthreads();                                   // this chunk is in place, the other buffer free
        if (more) fetch(k0 + KC);
        if (norm_row < 0) {
#pragma unroll
            for (int k = 0; k < KC; k += 2) {
                double2 x[RM], y[RN];
#pragma unroll
                for (int r = 0; r < RM; r++) x[r] = *(const double2*)&s[buf][ri + 4 * r][k];
#pragma unroll
                for (int c = 0; c < RN; c++) y[c] = *(const double2*)&s[buf][T::TI + cj + 8 * c][k];
#pragma unroll
                for (int r = 0; r < RM; r++)
#pragma unroll
                    for (int c = 0; c < RN; c++) {
                        acc[r][c] = __fma_rn(x[r].x, y[c].x, acc[r][c]);
                        acc[r][c] = __fma_rn(x[r].y, y[c].y, acc[r][c]);
                    }
            }
        } else if (norm_row < T::ROWS) {
#pragma unroll
            for (int k = 0; k < KC; k += 2) {
                const double2 x = *(const double2*)&s[buf][norm_row][k];
                nrm = __fma_rn(x.x, x.x, nrm);
                nrm = __fma_rn(x.y, x.y, nrm);
            }
        }
        if (more) put(buf ^ 1);
    }
    if (norm_row >= 0 && norm_row < T::ROWS) root[norm_row] = __dsqrt_rn(nrm);
    __syncthreads();
    if (norm_row >= 0) return;
#pragma unroll
    for (int r = 0; r < RM; r++) {
        const int i = i0 + ri + 4 * r;
        const double ra = root[ri + 4 * r];
#pragma unroll
        for (int c = 0; c < RN; c++) {
            const int j = j0 + cj + 8 * c;
            const double rb = root[T::TI + cj + 8 * c];
            // the square root of a squared norm is 0 exactly where the squared norm is
            const float q = (ra != 0.0 && rb != 0.0) ? (float)__ddiv_rn(acc[r][c], __dmul_rn(ra, rb)) : 0.0f;
            if (i < n && j < m) out[(size_t)i * pitch + j] = q;
        }
    }
}

template <int WR, int WC, int RM, int RN, int KC>
static cudaError_t launch_tile(const float* a, int n, const float* b, int m, float* out, size_t pitch, cudaStream_t s)
{
    using T = CosTile<WR, WC, RM, RN, KC>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((m + T::TJ - 1) / T::TJ, (n + T::TI - 1) / T::TI);
    cfg.blockDim = dim3(T::THREADS);
    cfg.stream = s;
    return cudaLaunchKernelEx(&cfg, cos_sim_matrix_kernel<WR, WC, RM, RN, KC>, a, n, b, m, out, pitch);
}

// Tiles of 16 x 16, 32 x 32 or 64 x 64 outputs: a larger one reads less shared memory per FMA and takes longer by itself.  A
// launch's time is close to fixed + wave x ceil(blocks / SMs) for each of them, with the constants below (us, fitted to
// 1 .. 1024 x 100 .. 10000: within 6 % of every time measured), and the least of the three is taken.
static cudaError_t launch_matrix(const float* a, int n, const float* b, int m, float* out, size_t pitch, int n_sm, cudaStream_t s)
{
    auto estimate = [&](int tile, double fixed, double wave) {
        const long long blocks = (long long)((n + tile - 1) / tile) * ((m + tile - 1) / tile);
        return fixed + wave * (double)((blocks + n_sm - 1) / n_sm);
    };
    const double t16 = estimate(16, 4.0, 8.2), t32 = estimate(32, 6.0, 15.7), t64 = estimate(64, 1.0, 46.0);
    if (t16 <= t32 && t16 <= t64) return launch_tile<4, 2, 1, 1, 64>(a, n, b, m, out, pitch, s);
    if (t32 <= t64) return launch_tile<4, 2, 2, 2, 32>(a, n, b, m, out, pitch, s);
    return launch_tile<4, 2, 4, 4, 16>(a, n, b, m, out, pitch, s);
}

// One call works in slices of at most CS_MAX_N x CS_MAX_M pairs, so the workspace a context keeps is bounded
// (4 + 8 + 32 MB) whatever the matrix.
#define CS_MAX_N 2048
#define CS_MAX_M 4096

static bool beyond_one_slice(int n, int m) { return n > CS_MAX_N || m > CS_MAX_M; }

// A result that takes the place of an input: every row has to be read before the first result is written.
static bool written_over(const float* out, int n, int m, const float* in, int rows)
{
    const uintptr_t o = (uintptr_t)out, i = (uintptr_t)in;
    return o < i + (size_t)rows * CS_DIM * sizeof(float) && i < o + (size_t)n * m * sizeof(float);
}

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

int CosWorkspace::run(int device, const float* ha, int n, const float* hb, int m, float* hout)
{
    const bool whole = written_over(hout, n, m, ha, n) || written_over(hout, n, m, hb, m);
    const int sn = whole ? n : std::min(n, CS_MAX_N), sm = whole ? m : std::min(m, CS_MAX_M);
    if ((!stream && cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking) != cudaSuccess) ||
        !grow(&a, &cap_a, (size_t)sn * CS_DIM) || !grow(&b, &cap_b, (size_t)sm * CS_DIM) || !grow(&out, &cap_out, (size_t)sn * sm)) {
        ffcu_set_error("ffcu_cos_sim_matrix: device allocation failed");
        cudaGetLastError();
        return -2;
    }
    int n_sm = 0;
    if (cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n_sm < 1) n_sm = 148;
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < n && e == cudaSuccess; i += sn) {
        const int cn = std::min(sn, n - i);
        e = cudaMemcpyAsync(a, ha + (size_t)i * CS_DIM, (size_t)cn * CS_DIM * 4, cudaMemcpyHostToDevice, stream);
        for (int j = 0; j < m && e == cudaSuccess; j += sm) {
            const int cm = std::min(sm, m - j);
            e = cudaMemcpyAsync(b, hb + (size_t)j * CS_DIM, (size_t)cm * CS_DIM * 4, cudaMemcpyHostToDevice, stream);
            if (e != cudaSuccess) break;
            // (the launch's own result: the thread's last error may be one that the caller has left there)
            e = launch_matrix(a, cn, b, cm, out, (size_t)cm, n_sm, stream);
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
    const int rc = w.run(device, a, n, b, m, out);
    w.release();
    return rc;
}

// The same through a workspace that its owner keeps.  Calls from several threads each go through: one takes the
// workspace, the others make their own for the call; so does a call that cannot go in slices, which the bound is for.
int CosWorkspace::call(int device, const float* ha, int n, const float* hb, int m, float* hout)
{
    if (!ha || !hb || !hout || n < 1 || m < 1) { ffcu_set_error("ffcu_cos_sim_matrix: bad arguments"); return -1; }
    if (beyond_one_slice(n, m) && (written_over(hout, n, m, ha, n) || written_over(hout, n, m, hb, m)))
        return ffcu_cos_sim_matrix(device, ha, n, hb, m, hout);
    if (!mu.try_lock()) return ffcu_cos_sim_matrix(device, ha, n, hb, m, hout);
    int rc = cudaSetDevice(device) == cudaSuccess ? 0 : -100;
    if (rc) { ffcu_set_error("cudaSetDevice(%d) failed", device); cudaGetLastError(); }
    else rc = run(device, ha, n, hb, m, hout);
    mu.unlock();
    return rc;
}
