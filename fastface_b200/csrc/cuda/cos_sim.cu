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
// 128 x 1000 51.4 | 61.6 | 22.6, 256 x 1000 82 | 72 | 37, 1024 x 1000 287 | 119 | 95, 1024 x 10000 2656 | 884 | 779.
#include "ffcu_internal.cuh"
#include "cos_sim.cuh"
#include "../host/ff_copy.h"

#include <stdint.h>
#include <string.h>
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

// One call works in slices of at most CS_MAX_N rows of `a` and CS_MAX_M of `b`, and a launch gives at most CS_MAX_OUT results,
// so the workspace a context keeps is bounded (4 + 32 + 2 x 10 MB on the device, 8 MB page-locked) whatever the matrix.  The plain
// way, which has no copy beside the kernel that more launches would help, takes CS_MAX_N x CS_PLAIN_M pairs at once (the kept result
// then up to 32 MB): in launches of CS_MAX_OUT, each with a copy of its own, 2000 x 4096 took 7.0 ms instead of 5.6, 2048 x 1400 over
// an input, which a kept workspace did not serve then, 3.6 instead of 1.5.
#define CS_MAX_N 2048
#define CS_MAX_M 16384
#define CS_PLAIN_M 4096
#define CS_MAX_OUT ((size_t)10 << 18)

static bool beyond_one_slice(int n, int m) { return n > CS_MAX_N || m > CS_PLAIN_M; }

// Rows and columns of the plain way's launches.
static void plain_slice(int n, int m, bool whole, int* sn, int* sm)
{
    *sn = whole ? n : std::min(n, CS_MAX_N);
    *sm = whole ? m : std::min(m, CS_PLAIN_M);
}

// Launches it makes for an n x m matrix, over an input or not.
extern "C" long long ffcu_test_cos_plain_launches(int n, int m, int over)
{
    int sn, sm;
    plain_slice(n, m, over != 0, &sn, &sm);
    return (long long)((n + sn - 1) / sn) * ((m + sm - 1) / sm);
}

// A result that takes the place of an input: every row has to be read before the first result is written.
static bool written_over(const float* out, int n, int m, const float* in, int rows)
{
    const uintptr_t o = (uintptr_t)out, i = (uintptr_t)in;
    return o < i + (size_t)rows * CS_DIM * sizeof(float) && i < o + (size_t)n * m * sizeof(float);
}

void CosWorkspace::release()
{
    cudaFree(a); cudaFree(b); cudaFree(out);
    for (cudaStream_t* s : {&stream, &s_in, &s_out}) { if (*s) cudaStreamDestroy(*s); *s = nullptr; }
    for (int k = 0; k < CS_PIECES; k++) for (cudaEvent_t* e : {&ev_in[k], &ev_out[k]}) { if (*e) cudaEventDestroy(*e); *e = nullptr; }
    for (cudaEvent_t* e : {&ev_uploaded, &ev_done[0], &ev_done[1]}) { if (*e) cudaEventDestroy(*e); *e = nullptr; }
    if (pin_in) cudaFreeHost(pin_in);
    if (pin_out) cudaFreeHost(pin_out);
    ff_copy_pool_destroy(pool);
    pin_in = pin_out = nullptr; pool = nullptr; tried = false; pieces_in = 0;
    a = b = out = nullptr; cap_a = cap_b = cap_out = 0;
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

static int device_sms(int device)
{
    int n_sm = 0;
    if (cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n_sm < 1) n_sm = 148;
    return n_sm;
}

// The plain way: a workspace of the call's own, or a result that takes the place of an input.
int CosWorkspace::run(int device, const float* ha, int n, const float* hb, int m, float* hout)
{
    const bool whole = written_over(hout, n, m, ha, n) || written_over(hout, n, m, hb, m);
    int sn, sm;
    plain_slice(n, m, whole, &sn, &sm);
    if ((!stream && cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking) != cudaSuccess) ||
        !grow(&a, &cap_a, (size_t)sn * CS_DIM) || !grow(&b, &cap_b, (size_t)sm * CS_DIM) || !grow(&out, &cap_out, (size_t)sn * sm)) {
        ffcu_set_error("ffcu_cos_sim_matrix: device allocation failed");
        cudaGetLastError();
        return -2;
    }
    const int n_sm = device_sms(device);
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

// ---------------------------------------------------------------------------
// A kept workspace: copies shared by several threads through page-locked pieces, one way beside the other and beside the
// kernels.  The driver's own staging of pageable memory is one thread (12 GB/s) and blocks the caller: of the 647 us of a
// 1024 x 1024 call the kernel was 95.  Pageable calls, driver's staging -> this, us: 1 x 100 56 -> 53, 16 x 300 79 -> 63, 1 x 1000
// 169 -> 108, 64 x 1000 207 -> 138, 1 x 10000 1220 -> 560, 128 x 10000 1622 -> 798, 1024 x 1000 597 -> 338, 1024 x 10000 9697 -> 4819
// (the caller's untouched pages); 1 ... 1024 x 100 ... 10000, 54 sizes: none slower.
// ---------------------------------------------------------------------------
bool CosWorkspace::pipeline_ready()
{
    if (tried) return pin_out != nullptr;
    tried = true;
    bool ok = true;
    for (cudaStream_t* s : {&stream, &s_in, &s_out}) if (!*s) ok = ok && cudaStreamCreateWithFlags(s, cudaStreamNonBlocking) == cudaSuccess;
    for (int k = 0; k < CS_PIECES; k++)
        for (cudaEvent_t* e : {&ev_in[k], &ev_out[k]}) ok = ok && cudaEventCreateWithFlags(e, cudaEventDisableTiming) == cudaSuccess;
    for (cudaEvent_t* e : {&ev_uploaded, &ev_done[0], &ev_done[1]}) ok = ok && cudaEventCreateWithFlags(e, cudaEventDisableTiming) == cudaSuccess;
    ok = ok && (pin_in = ffcu_stage_alloc(CS_PIECES * CS_PIECE)) && (pin_out = ffcu_stage_alloc(CS_PIECES * CS_PIECE));
    if (!ok) {
        cudaGetLastError();
        if (pin_in) cudaFreeHost(pin_in);
        if (pin_out) cudaFreeHost(pin_out);
        pin_in = pin_out = nullptr;
        return false;
    }
    pool = ff_copy_pool_create(3);                    // NULL: the caller's thread copies alone
    return true;
}

// Host -> device on s_in; a pageable source has been read when this returns.
cudaError_t CosWorkspace::upload(float* dst, const float* src, size_t bytes, bool staged)
{
    if (!staged) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s_in);
    cudaError_t e = cudaSuccess;
    for (size_t o = 0; o < bytes && e == cudaSuccess; o += CS_PIECE, pieces_in++) {
        const size_t nb = std::min(CS_PIECE, bytes - o);
        const unsigned k = pieces_in % CS_PIECES;
        if (pieces_in >= CS_PIECES) e = cudaEventSynchronize(ev_in[k]);        // the slot's last copy has left it
        if (e != cudaSuccess) break;
        ff_copy(pool, pin_in + k * CS_PIECE, (const char*)src + o, nb, 1);
        e = cudaMemcpyAsync((char*)dst + o, pin_in + k * CS_PIECE, nb, cudaMemcpyHostToDevice, s_in);
        if (e == cudaSuccess) e = cudaEventRecord(ev_in[k], s_in);
    }
    return e;
}

// rows x cols results at src, complete with event `done`, -> host rows `pitch` floats apart, by way of s_out.
cudaError_t CosWorkspace::deliver(float* hout, size_t pitch, const float* src, int rows, int cols, bool staged, cudaEvent_t done)
{
    cudaError_t e = cudaStreamWaitEvent(s_out, done, 0);
    if (e != cudaSuccess) return e;
    if (!staged)
        return (size_t)cols == pitch ? cudaMemcpyAsync(hout, src, (size_t)rows * cols * 4, cudaMemcpyDeviceToHost, s_out)
                                     : cudaMemcpy2DAsync(hout, pitch * 4, src, (size_t)cols * 4, (size_t)cols * 4, rows, cudaMemcpyDeviceToHost, s_out);
    const size_t total = (size_t)rows * cols * 4, n = (total + CS_PIECE - 1) / CS_PIECE;
    auto fetch = [&](size_t p) {
        const size_t nb = std::min(CS_PIECE, total - p * CS_PIECE);
        cudaError_t r = cudaMemcpyAsync(pin_out + p % CS_PIECES * CS_PIECE, (const char*)src + p * CS_PIECE, nb, cudaMemcpyDeviceToHost, s_out);
        return r == cudaSuccess ? cudaEventRecord(ev_out[p % CS_PIECES], s_out) : r;
    };
    for (size_t p = 0; p < std::min<size_t>(n, CS_PIECES) && e == cudaSuccess; p++) e = fetch(p);
    for (size_t p = 0; p < n && e == cudaSuccess; p++) {
        e = cudaEventSynchronize(ev_out[p % CS_PIECES]);
        if (e != cudaSuccess) break;
        const size_t o = p * CS_PIECE, nb = std::min(CS_PIECE, total - o), line = (size_t)cols * 4;
        const char* from = pin_out + p % CS_PIECES * CS_PIECE;
        if ((size_t)cols == pitch) ff_copy(pool, (char*)hout + o, from, nb, 0);
        else
            for (size_t x = o; x < o + nb; ) {                                  // the rows of a column slice, a piece's first and last in parts
                const size_t row = x / line, at = x % line, part = std::min(line - at, o + nb - x);
                memcpy((char*)(hout + row * pitch) + at, from + (x - o), part);
                x += part;
            }
        if (p + CS_PIECES < n) e = fetch(p + CS_PIECES);
    }
    return e;
}

// Rows of a launch for m columns: whole 64-row tiles that fill the SMs (at least 85 % of the launch's last wave), as few as
// that takes, so that the results of one launch are on their way while the next one runs; at most CS_MAX_OUT results.
static int launch_rows(int m, int n_sm)
{
    const int tiles = (m + 63) / 64;
    const int most = (int)std::max<size_t>(CS_MAX_OUT / ((size_t)64 * m), 1);
    int best = 1;
    double best_fill = 0.0;
    for (int k = 1; k <= most && best_fill < 0.85; k++) {
        const long long blocks = (long long)k * tiles, waves = (blocks + n_sm - 1) / n_sm;
        const double fill = (double)blocks / (double)(waves * n_sm);
        if (fill > best_fill) { best = k; best_fill = fill; }
    }
    return 64 * best;
}

int CosWorkspace::run_pipeline(int n_sm, const float* ha, int n, const float* hb, int m, float* hout, bool in_a, bool in_b, bool out_staged)
{
    const size_t in_bytes = (size_t)(n + m) * CS_DIM * 4, out_bytes = (size_t)n * m * 4;
    pieces_in = 0;                                    // the last call has waited for its copies: the ring is free (and the count cannot run over)
    if (in_a && in_b && out_staged && in_bytes <= CS_PIECE && out_bytes <= CS_PIECE) {
        // a small matrix: both inputs in one copy, everything in order on one stream (1 x 100 / 1 x 300: 63 / 77 -> 53 / 60 us)
        if (!grow(&b, &cap_b, (size_t)(n + m) * CS_DIM) || !grow(&out, &cap_out, (size_t)n * m)) {
            ffcu_set_error("ffcu_cos_sim_matrix: device allocation failed");
            cudaGetLastError();
            return -2;
        }
        ff_copy(pool, pin_in, hb, (size_t)m * CS_DIM * 4, 1);
        ff_copy(pool, pin_in + (size_t)m * CS_DIM * 4, ha, (size_t)n * CS_DIM * 4, 1);
        cudaError_t e = cudaMemcpyAsync(b, pin_in, in_bytes, cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess) e = launch_matrix(b + (size_t)m * CS_DIM, n, b, m, out, (size_t)m, n_sm, stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(pin_out, out, out_bytes, cudaMemcpyDeviceToHost, stream);
        const cudaError_t e2 = cudaStreamSynchronize(stream);
        if (e == cudaSuccess) e = e2;
        if (e != cudaSuccess) { ffcu_set_error("ffcu_cos_sim_matrix: %s", cudaGetErrorString(e)); return -100; }
        ff_copy(pool, hout, pin_out, out_bytes, 0);
        return 0;
    }
    const int sn = std::min(n, CS_MAX_N), sm = std::min(m, CS_MAX_M);
    const int step = std::min(sn, launch_rows(sm, n_sm));
    const size_t slot = (size_t)step * sm;
    cudaError_t e = cudaSuccess;
    int rc = 0;
    if (!grow(&a, &cap_a, (size_t)sn * CS_DIM) || !grow(&b, &cap_b, (size_t)sm * CS_DIM) ||
        !grow(&out, &cap_out, slot * (step < n || sm < m ? 2 : 1))) {
        ffcu_set_error("ffcu_cos_sim_matrix: device allocation failed");
        cudaGetLastError();
        return -2;
    }
    if (!in_a && !in_b && !out_staged && n <= step && m <= sm) {
        // page-locked arrays and one launch: nothing runs beside anything, and the other streams only cost their hops (1 x 100 / 16 x 300 / 64 x 1000 /
        // 128 x 1000 / 512 x 1000: 46.9 / 54.4 / 92.7 / 108.1 / 173.6 -> 48.1 / 49.0 / 93.1 / 100.1 / 173.5 us)
        e = cudaMemcpyAsync(a, ha, (size_t)n * CS_DIM * 4, cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(b, hb, (size_t)m * CS_DIM * 4, cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess) e = launch_matrix(a, n, b, m, out, (size_t)m, n_sm, stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(hout, out, (size_t)n * m * 4, cudaMemcpyDeviceToHost, stream);
        const cudaError_t e2 = cudaStreamSynchronize(stream);
        if (e == cudaSuccess) e = e2;
        if (e != cudaSuccess) { ffcu_set_error("ffcu_cos_sim_matrix: %s", cudaGetErrorString(e)); return -100; }
        return 0;
    }
    struct { float* to; const float* from; int rows, cols; } last = {nullptr, nullptr, 0, 0};      // launched, not delivered
    int k = 0;                                        // launches so far
    auto flush = [&]() {
        if (e == cudaSuccess && last.to) e = deliver(last.to, (size_t)m, last.from, last.rows, last.cols, out_staged, ev_done[(k - 1) & 1]);
        last.to = nullptr;
    };
    for (int i0 = 0; i0 < n && e == cudaSuccess; i0 += sn) {
        const int cn = std::min(sn, n - i0);
        for (int j = 0; j < m && e == cudaSuccess; j += sm) {
            const int cm = std::min(sm, m - j);
            if (k) e = cudaStreamWaitEvent(s_in, ev_done[(k - 1) & 1], 0);      // what the earlier launches read is replaced
            if (e == cudaSuccess) e = upload(b, hb + (size_t)j * CS_DIM, (size_t)cm * CS_DIM * 4, in_b);
            for (int i = 0; i < cn && e == cudaSuccess; i += step) {
                const int rows = std::min(step, cn - i);
                if (j == 0) e = upload(a + (size_t)i * CS_DIM, ha + (size_t)(i0 + i) * CS_DIM, (size_t)rows * CS_DIM * 4, in_a);
                if (e == cudaSuccess) e = cudaEventRecord(ev_uploaded, s_in);
                if (e == cudaSuccess) e = cudaStreamWaitEvent(stream, ev_uploaded, 0);
                float* to = out + (size_t)(k & 1) * slot;
                if (e == cudaSuccess && !out_staged && k >= 2) e = cudaStreamSynchronize(s_out);    // the slot's copy has left it (a staged one has been waited for)
                if (e == cudaSuccess) e = launch_matrix(a + (size_t)i * CS_DIM, rows, b, cm, to, (size_t)cm, n_sm, stream);
                if (e == cudaSuccess) e = cudaEventRecord(ev_done[k & 1], stream);
                flush();                              // the launch before, while this one runs
                last = {hout + (size_t)(i0 + i) * m + j, to, rows, cm};
                k++;
            }
        }
    }
    flush();
    for (cudaStream_t s : {s_in, stream, s_out}) {
        const cudaError_t e2 = cudaStreamSynchronize(s);
        if (e == cudaSuccess) e = e2;
    }
    if (e != cudaSuccess) { ffcu_set_error("ffcu_cos_sim_matrix: %s", cudaGetErrorString(e)); rc = -100; }
    return rc;
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
    const bool over = written_over(hout, n, m, ha, n) || written_over(hout, n, m, hb, m);
    if (beyond_one_slice(n, m) && over) return ffcu_cos_sim_matrix(device, ha, n, hb, m, hout);
    if (!mu.try_lock()) return ffcu_cos_sim_matrix(device, ha, n, hb, m, hout);
    int rc = cudaSetDevice(device) == cudaSuccess ? 0 : -100;
    if (rc) { ffcu_set_error("cudaSetDevice(%d) failed", device); cudaGetLastError(); }
    else if (over || !pipeline_ready()) rc = run(device, ha, n, hb, m, hout);
    else rc = run_pipeline(device_sms(device), ha, n, hb, m, hout, ffcu_is_pageable(ha, (size_t)n * CS_DIM * 4),
                           ffcu_is_pageable(hb, (size_t)m * CS_DIM * 4), ffcu_is_pageable(hout, (size_t)n * m * 4));
    mu.unlock();
    return rc;
}
