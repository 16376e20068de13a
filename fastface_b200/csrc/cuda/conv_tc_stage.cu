// conv_tc_stage.cu -- small batches: the 14x14 stage (a run of 3x3 stride-1 256 -> 256 convolutions) in ONE launch, a cluster of
// eight or four CTAs per face, activations in shared memory.
//
// The operands as in conv_tc_face.cu (weights are the MMA's 128 rows, a row of the face 16 of its columns), but every CTA issues
// its own MMAs: a cluster is 2 halves of the output channels x R tiles of the face's rows (R = 4: 4, 4, 3 and 3 rows, 64 columns;
// R = 2: 7 rows, 112 columns).  A CTA holds, for both halves' channels, its rows and one above and below, in two buffers that
// take turns.  Its epilogue writes its 128 channels of its rows into its own next buffer, bytewise, and sends the rows from there by
// bulk copies: all of them to the CTA with the other channels of the same rows, the first and the last to both CTAs of the
// neighbouring rows.
//
// Bound: latency.  What passes between shared memories goes at 20 B per cycle and CTA whatever instruction sends it (measured:
// 8 KB to 1 / 2 / 4 / 8 CTAs of a cluster of eight 710 / 1110 / 1920 / 3550 cycles by 16-byte st.async, 810 / 1210 / 2005 / 3790 by bulk copies), so the split
// is the one that sends least: 16 KB per CTA and layer instead of 36 KB for 2 row tiles x 4 channel tiles (conv_tc_chain.cu).
// Forward of 1 / 4 / 8 / 15 faces, that chain -> clusters of eight: 273 / 287 / 309 / 349 -> 230 / 249 / 267 / 304 us; of 16 / 17 / 24 / 33
// faces, its wide form -> clusters of four: 409 / 413 / 445 / 487 -> 357 / 361 / 396 / 435 us (14x14 layers 5.1 -> 3.5 and 7 -> 5 us).
//
// Replaces, per layer, what conv_tc_kernel does (reference kernels/conv2d_nhwc.c:179-220, kernels/int8_epilogue.c:25-112,
// :253-318); same arithmetic, same bytes.
#include "conv_tc_face.cuh"

namespace {

template <int R>
struct Stage {
    static constexpr int ROWS = R == 4 ? 4 : 7;              // rows of a tile (R = 4: the last two have three)
    static constexpr int PER_GROUP = (ROWS + 3) / 4;         // rows of an epilogue group of four warps
    static constexpr int N = ROWS * 16;
    static constexpr int PLANE_BYTES = (ROWS + 2) * 2048;
    static constexpr int ACT_BYTES = 2 * PLANE_BYTES;
    static constexpr int STEP_BYTES = 2 * 128 * 128;         // one filter tap: 128 output channels x 256 input channels
    static constexpr int STAGES = R == 4 ? 4 : 3;
    static constexpr int OFF_LUT = 2 * ACT_BYTES;
    static constexpr int OFF_RING = OFF_LUT + FACE_LUT_BYTES;
    static constexpr int OFF_SH = OFF_RING + STAGES * STEP_BYTES;
    static constexpr uint32_t TMEM_COLS = R == 4 ? 64 : 128;
    static_assert(OFF_RING % 1024 == 0 && ACT_BYTES % 1024 == 0, "swizzle atoms");
    __device__ static int first_row(int t) { return R == 4 ? (t < 2 ? 4 * t : 8 + 3 * (t - 2)) : 7 * t; }
    __device__ static int rows(int t) { return R == 4 ? (t < 2 ? 4 : 3) : 7; }
};

struct StageShared {
    uint64_t full[4], empty[4];
    uint64_t a0_full;             // the first input has landed, and the padding's zeros in both buffers
    uint64_t act_full[2];         // buffer b holds the next layer's input: own rows (sixteen warps), and the bytes that come
    uint64_t acc_full;
    uint64_t lut_full, lut_empty;
    uint32_t tmem_base;
    int abort_flag;
};

// One layer.  RESBN: residual and fused BN (else PReLU); LAST: results go to global memory as NHWC.
template <bool CONTRACT, int R, bool RESBN, bool LAST>
__device__ __forceinline__ void stage_epilogue(uint8_t* smem, StageShared* sh, const FaceLayer* cl, const float4& k, int L, int rank, int q, int g,
                                               int lane, uint32_t lut_lo, uint32_t lut_hi, int face, int8_t* kept, uint32_t tmem_base,
                                               uint32_t lut_parity, volatile int* abort_flag, const FaceParams& p, bool& ok)
{
    using S = Stage<R>;
    constexpr int PG = S::PER_GROUP;
    const int h = rank & 1, t = rank >> 1, ch = q * 32 + lane;
    const int n_rows = S::rows(t), r0 = S::first_row(t);
    const int mine = n_rows - g * PG < PG ? n_rows - g * PG : PG;          // rows of this warp's group: r0 + g * PG ..  (may be <= 0)
    const size_t px0 = ((size_t)face * 196 + (size_t)(r0 + g * PG) * 14) * FACE_C + h * 128 + ch;
    uint32_t rw[4 * PG];
#pragma unroll
    for (int i = 0; i < 4 * PG; i++) rw[i] = 0;
    if (RESBN && ok) {
        const int8_t* res = cl->res;
#pragma unroll
        for (int r = 0; r < PG; r++) {
            if (r >= mine) break;
            if (res) {
#pragma unroll
                for (int c = 0; c < 14; c++) {
                    uint32_t b;
                    asm volatile("ld.global.u8 %0, [%1];" : "=r"(b) : "l"(res + px0 + (size_t)(r * 14 + c) * FACE_C));
                    rw[4 * r + c / 4] |= b << (8 * (c & 3));
                }
            } else
                asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(rw[4 * r]), "=r"(rw[4 * r + 1]), "=r"(rw[4 * r + 2]), "=r"(rw[4 * r + 3])
                             : "l"(kept + r * (FACE_C * 16)));
        }
    }
    if (RESBN && ok) ok = mbar_wait(smem_u32(&sh->lut_full), lut_parity, abort_flag, p.err, FFCU_ERR_TMA_TIMEOUT, p.wait_cycles);
    if (ok) ok = mbar_wait(smem_u32(&sh->acc_full), (uint32_t)L & 1, abort_flag, p.err, FFCU_ERR_EPI_TIMEOUT, p.wait_cycles);
    tc_fence_after();
    const uint8_t* lut = smem + S::OFF_LUT;
    const uint32_t taddr = tmem_base + (uint32_t)(g * PG * 16) + ((uint32_t)(q * 32) << 16);
    const uint32_t s_plane = smem_u32(smem) + (uint32_t)(((L + 1) & 1) * S::ACT_BYTES + h * S::PLANE_BYTES);
    const uint32_t s_rows = s_plane + (uint32_t)((g * PG + 1) * 2048);     // the group's rows in the next input
    if (ok && mine > 0) {
        FaceDst d;
        if (LAST) d.g = cl->out2 + px0;
        else {
#pragma unroll
            for (int i = 0; i < 8; i++) d.ad[i] = (s_rows + (uint32_t)ch) ^ (uint32_t)(i << 4);
        }
        int va[16], vb[16];
        tmem_ld16_issue(taddr, va);
        tmem_ld_wait(va);
        if (PG == 2 && mine > 1) tmem_ld16_issue(taddr + 16, vb);
        face_cols<CONTRACT, RESBN, LAST, 0, 8, 0>(va, rw, k, lut, lut_lo, lut_hi, d);
        face_cols<CONTRACT, RESBN, LAST, 8, 14, 0>(va + 8, rw + 2, k, lut, lut_lo, lut_hi, d);
        if (PG == 2 && mine > 1) {
            tmem_ld_wait(vb);
            face_cols<CONTRACT, RESBN, LAST, 0, 8, 1>(vb, rw + (PG == 2 ? 4 : 0), k, lut, lut_lo, lut_hi, d);
            face_cols<CONTRACT, RESBN, LAST, 8, 14, 1>(vb + 8, rw + (PG == 2 ? 6 : 0), k, lut, lut_lo, lut_hi, d);
        }
    }
    if (!LAST) {
        // Every warp comes here whatever its ok flag: none may be left waiting.  (What the warps have read of the accumulator
        // counts with the same arrival.)
        fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && ok) mbar_arrive(smem_u32(&sh->act_full[(L + 1) & 1]));
        asm volatile("bar.sync %0, 128;" ::"r"(2 + g) : "memory");
        if (ok && lane == 0 && mine > 0) {
            const uint32_t bar = smem_u32(&sh->act_full[(L + 1) & 1]);
            if (q == 0) bulk_send(map_to_cta(s_rows, (uint32_t)rank ^ 1u), s_rows, (uint32_t)(mine * 2048), map_to_cta(bar, (uint32_t)rank ^ 1u));
            else if (q < 3) {
                // the first row is the row below the tile above's, the last one the row above the tile below's
                const uint32_t other = q == 1 ? 0u : 1u;
                if (g == 0 && t > 0) {
                    const uint32_t to = ((uint32_t)rank - 2u) ^ other;
                    bulk_send(map_to_cta(s_plane + (uint32_t)((S::rows(t - 1) + 1) * 2048), to), s_rows, 2048, map_to_cta(bar, to));
                }
                if (g == (n_rows - 1) / PG && t < R - 1) {
                    const uint32_t to = ((uint32_t)rank + 2u) ^ other;
                    bulk_send(map_to_cta(s_plane, to), s_plane + (uint32_t)(n_rows * 2048), 2048, map_to_cta(bar, to));
                }
            }
        }
    }
    if (ok && RESBN && !LAST) {
#pragma unroll
        for (int r = 0; r < PG; r++)
            if (r < mine)
                asm volatile("st.global.v4.b32 [%0], {%1, %2, %3, %4};" ::"l"(kept + r * (FACE_C * 16)), "r"(rw[4 * r]), "r"(rw[4 * r + 1]), "r"(rw[4 * r + 2]), "r"(rw[4 * r + 3]) : "memory");
    }
    if (ok && LAST) {
        int8_t* out = cl->out + px0;
#pragma unroll
        for (int r = 0; r < PG; r++)
            if (r < mine) {
#pragma unroll
                for (int c = 0; c < 14; c++) out[(r * 14 + c) * FACE_C] = (int8_t)(rw[4 * r + c / 4] >> (8 * (c & 3)));
            }
    }
}

template <bool CONTRACT, int R>
__global__ void __launch_bounds__(TC_THREADS, 1)
conv_stage_kernel(const __grid_constant__ CUtensorMap mapA, const FaceParams p)
{
    using S = Stage<R>;
    extern __shared__ __align__(1024) uint8_t smem[];
    StageShared* sh = (StageShared*)(smem + S::OFF_SH);
    if (smem_u32(smem) & 1023) {                              // the swizzle atoms' alignment, as the declaration asks for it
        if (threadIdx.x == 0) atomicCAS(p.err, 0, FFCU_ERR_TMA_TIMEOUT);
        return;
    }
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int rank = (int)cluster_ctarank();
    const int cluster = (int)blockIdx.x / (2 * R), face = p.face0 + cluster;
    const int h = rank & 1, t = rank >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S::STAGES; s++) { mbar_init(smem_u32(&sh->full[s]), 1); mbar_init(smem_u32(&sh->empty[s]), 1); }
        mbar_init(smem_u32(&sh->a0_full), 1);
        for (int b = 0; b < 2; b++) mbar_init(smem_u32(&sh->act_full[b]), 17);          // the epilogue's warps, one arming arrival
        mbar_init(smem_u32(&sh->acc_full), 1);
        mbar_init(smem_u32(&sh->lut_full), 1);
        mbar_init(smem_u32(&sh->lut_empty), 16);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == TC_ISSUER_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&sh->tmem_base)), "r"(S::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                       // the peers' barriers are initialised
    tc_fence_after();
    const uint32_t tmem_base = sh->tmem_base;
    volatile int* abort_flag = &sh->abort_flag;
    const uint32_t s0 = smem_u32(smem);

    if (warp == TC_PRODUCER_WARP) {
        // Weight producer: a step is one filter tap, two boxes (lane i: input channels 128 i ..)
        int stage = 0, gs = 0; uint32_t phase = 0;
        bool ok = true;
#pragma unroll 1
        for (int L = 0; L < p.n_layers && ok; L++) {
            const CUtensorMap* map = &p.layers[L].mapB;
            if (lane < 2) asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
#pragma unroll 1
            for (int tap = 0; tap < 9; tap++, gs++) {
                ok = mbar_wait(smem_u32(&sh->empty[stage]), phase ^ 1, abort_flag, p.err, FFCU_ERR_EMPTY_TIMEOUT, p.wait_cycles);
                if (!ok) break;
                if (lane == 0) mbar_expect_tx(smem_u32(&sh->full[stage]), S::STEP_BYTES);
                __syncwarp();
                // (drop_step: the timeout test's launch, CTA 0 leaves out this step)
                if (lane < 2 && (gs != p.drop_step || rank != 0))
                    tma_load_4d(s0 + S::OFF_RING + stage * S::STEP_BYTES + lane * (128 * 128), map, smem_u32(&sh->full[stage]), tap * FACE_C + lane * 128, h * 128, 0, 0);
                if (++stage == S::STAGES) { stage = 0; phase ^= 1; }
            }
        }
    } else if (warp == TC_ISSUER_WARP) {
        if (tc_elect_one()) {
            constexpr uint32_t IDESC = idesc_i8(S::N);
            const uint32_t full0 = smem_u32(&sh->full[0]), empty0 = smem_u32(&sh->empty[0]);
            const uint64_t da0 = smem_desc<128>(s0 + S::OFF_RING);
            // what this CTA receives of each layer: its rows' other channels, and the rows above and below
            const uint32_t in_bytes = (uint32_t)(S::rows(t) * 2048 + (t > 0 ? 4096 : 0) + (t < R - 1 ? 4096 : 0));
            int stage = 0; uint32_t phase = 0, ready = 0;
            bool ok = true;
#pragma unroll 1
            for (int L = 0; L < p.n_layers && ok; L++) {
                const int buf = L & 1;
                // (bytes that land before this only drive the count negative: the phase needs this arrival)
                if (L + 1 < p.n_layers) mbar_expect_tx(smem_u32(&sh->act_full[buf ^ 1]), in_bytes);
                ok = L == 0 ? mbar_wait(smem_u32(&sh->a0_full), 0, abort_flag, p.err, FFCU_ERR_TMA_TIMEOUT, p.wait_cycles)
                            : mbar_wait_cluster(smem_u32(&sh->act_full[buf]), (uint32_t)((L - 1) >> 1) & 1, abort_flag, p.err, FFCU_ERR_TMA_TIMEOUT, p.wait_cycles);
                if (!ok) break;
                tc_fence_after();
                uint64_t db_row = smem_desc<128>(s0 + (uint32_t)(buf * S::ACT_BYTES));
                uint32_t first = 0;
#pragma unroll 1
                for (int kh = 0; kh < 3 && ok; kh++, db_row += 2048 / 16) {
#pragma unroll
                    for (int kw = 0; kw < 3; kw++) {
                        if (!ready) {
                            ok = mbar_wait(full0 + stage * 8, phase, abort_flag, p.err, FFCU_ERR_TMA_TIMEOUT, p.wait_cycles);
                            if (!ok) break;
                        }
                        int ns = stage + 1; uint32_t np = phase;
                        if (ns == S::STAGES) { ns = 0; np ^= 1; }
                        ready = mbar_test(full0 + ns * 8, np);                   // used next round
                        tc_fence_after();
                        const uint64_t da = da0 + (uint64_t)((uint32_t)(stage * S::STEP_BYTES) >> 4);
#pragma unroll
                        for (int pl = 0; pl < 2; pl++)
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                umma_i8(tmem_base, da + (uint64_t)(pl * (128 * 128 >> 4) + 2 * k), db_row + (uint64_t)(((kw * 128 + pl * S::PLANE_BYTES) >> 4) + 2 * k),
                                        IDESC, (kw | pl | k) ? 1u : first);
                        first = 1;
                        umma_commit(empty0 + stage * 8);
                        stage = ns; phase = np;
                    }
                }
                if (ok) umma_commit(smem_u32(&sh->acc_full));
            }
        }
    } else if (warp == TC_ISSUER2_WARP) {
        // The face's first input, into both buffers (of the second only the padding's zeros stay), and the fused BNs' byte tables
        if (tc_elect_one()) {
            tc_pdl_wait();
            mbar_expect_tx(smem_u32(&sh->a0_full), 2 * S::ACT_BYTES);
#pragma unroll
            for (int i = 0; i < 4; i++)
                tma_load_4d(s0 + i * S::PLANE_BYTES, &mapA, smem_u32(&sh->a0_full), (i & 1) * 128, -1, S::first_row(t) - 1, face);
            uint32_t lut_par = 0;
            bool ok = true;
#pragma unroll 1
            for (int L = 0; L < p.n_layers && ok; L++) {
                // (a layer at a time, so that a launch that hangs does so at the wait that is to blame)
                if (L) ok = mbar_wait(smem_u32(&sh->acc_full), (uint32_t)(L - 1) & 1, abort_flag, p.err, FFCU_ERR_EPI_TIMEOUT, p.wait_cycles);
                const uint8_t* lut = p.layers[L].lut;
                if (!lut || !ok) continue;
                ok = mbar_wait(smem_u32(&sh->lut_empty), lut_par ^ 1, abort_flag, p.err, FFCU_ERR_EMPTY_TIMEOUT, p.wait_cycles);
                lut_par ^= 1;
                if (!ok) break;
                mbar_expect_tx(smem_u32(&sh->lut_full), FACE_LUT_BYTES);
                bulk_load(s0 + S::OFF_LUT, lut + h * FACE_LUT_BYTES, FACE_LUT_BYTES, smem_u32(&sh->lut_full));
            }
        }
    } else {
        const int q = warp & 3, g = warp >> 2;
        const uint32_t lut_lo = (uint32_t)(lane * 4 + (q & 1) * 128) * 0x01010101u, lut_hi = (uint32_t)(q >> 1) * 0x01010101u;
        // a result that the next residual layer adds lies as its thread left it: a row of a channel in 16 bytes
        int8_t* kept = p.kept + (size_t)cluster * FACE_KEPT_BYTES + ((size_t)(S::first_row(t) + g * S::PER_GROUP) * FACE_C + h * 128 + q * 32 + lane) * 16;
        uint32_t lut_par = 0;
        bool ok = true;
        tc_pdl_wait();
#pragma unroll 1
        for (int L = 0; L < p.n_layers; L++) {
            const FaceLayer* cl = p.layers + L;
            const float4 k = __ldg(cl->tab + h * 128 + q * 32 + lane);
            const bool bn = cl->lut != nullptr;
            const bool last = L + 1 == p.n_layers;
            // (the next kernel not before: its CTAs would keep other contexts' kernels off the SMs this launch leaves free)
            if (last && warp == 0) tc_pdl_trigger();
            if (last)    stage_epilogue<CONTRACT, R, true, true>(smem, sh, cl, k, L, rank, q, g, lane, lut_lo, lut_hi, face, kept, tmem_base, lut_par, abort_flag, p, ok);
            else if (bn) stage_epilogue<CONTRACT, R, true, false>(smem, sh, cl, k, L, rank, q, g, lane, lut_lo, lut_hi, face, kept, tmem_base, lut_par, abort_flag, p, ok);
            else         stage_epilogue<CONTRACT, R, false, false>(smem, sh, cl, k, L, rank, q, g, lane, lut_lo, lut_hi, face, kept, tmem_base, lut_par, abort_flag, p, ok);
            if (bn) {
                lut_par ^= 1;
                __syncwarp();
                if (lane == 0) mbar_arrive_relaxed(smem_u32(&sh->lut_empty));
            }
        }
    }
    // teardown: nobody leaves before the whole cluster is here, so no CTA's memory is read or written after it has exited
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && threadIdx.x == 0) {
#pragma unroll 1
        for (int i = 0; i < 1000; i++) __nanosleep(1000);
    }
    __syncthreads();
    cluster_sync_all();
    if (warp == TC_ISSUER_WARP) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(S::TMEM_COLS) : "memory");
    }
}

template <int R>
constexpr int smem_bytes() { return Stage<R>::OFF_SH + (int)sizeof(StageShared); }

template <bool CONTRACT, int R>
int set_smem()
{
    static int done[64] = {};             // per device: the attribute belongs to the device's copy of the function
    int dev = 0;
    FFCU_CHECK(cudaGetDevice(&dev));
    if (!done[dev & 63]) {
        FFCU_CHECK(cudaFuncSetAttribute(conv_stage_kernel<CONTRACT, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<R>()));
        done[dev & 63] = 1;
    }
    return 0;
}

template <bool CONTRACT, int R>
int launch_stage(int faces, cudaStream_t s, const CUtensorMap& mapA, const FaceParams& prm)
{
    const int rc = set_smem<CONTRACT, R>();
    return rc != 0 ? rc : tc_launch_ex(conv_stage_kernel<CONTRACT, R>, 2 * R * faces, smem_bytes<R>(), s, 2 * R, mapA, prm);
}

template <int R>
int stage_clusters()
{
    if (set_smem<true, R>() != 0 || set_smem<false, R>() != 0) { cudaGetLastError(); return 0; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * R);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smem_bytes<R>();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * R; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, conv_stage_kernel<true, R>, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
    return n;
}

}  // namespace

int tc_launch_stage(int row_tiles, int mode, int faces, cudaStream_t s, const CUtensorMap& mapA, const FaceParams& prm)
{
    if (row_tiles == 4) return mode ? launch_stage<true, 4>(faces, s, mapA, prm) : launch_stage<false, 4>(faces, s, mapA, prm);
    return mode ? launch_stage<true, 2>(faces, s, mapA, prm) : launch_stage<false, 2>(faces, s, mapA, prm);
}

// How many clusters (two CTAs per row tile) the device holds at once.
int tc_stage_clusters(int row_tiles) { return row_tiles == 4 ? stage_clusters<4>() : stage_clusters<2>(); }
