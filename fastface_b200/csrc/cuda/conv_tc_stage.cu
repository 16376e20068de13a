// conv_tc_stage.cu -- small batches: a stage (a run of 3x3 stride-1 C -> C convolutions) in ONE launch, a cluster of two to eight
// CTAs per face, activations in shared memory: 128 channels on 28x28 maps, 256 on 14x14, 512 on 7x7.
//
// The operands as in conv_tc_face.cu (weights are the MMA's 128 rows, a row of the face 8, 16 or 32 of its columns), but every
// CTA issues its own MMAs: a cluster is C / 128 tiles of the output channels x R tiles of the face's rows, in two forms:
//
//     maps        few faces                                  while the device holds that many clusters
//     28x28       R = 7, 4 rows, 128 columns; 7 CTAs         R = 4, 7 rows, 224 columns; 4 CTAs
//     14x14       R = 4, 4 / 3 rows, 64 columns; 8 CTAs      R = 2, 7 rows, 112 columns; 4 CTAs
//     7x7         R = 2, 4 / 3 rows, 32 columns; 8 CTAs      R = 1, 7 rows, 64 columns; 4 CTAs
//
// From 49 to 74 faces the 28x28 stage also goes in clusters of two: 14 rows a CTA, as two accumulators of 224 columns from the same
// weights, emptied one after the other (forward of 64 / 74 faces 572 / 636 -> 564 / 626 us).
// On 7x7 maps a cluster of four also takes two faces at once (128 columns), one under the other with a row of zeros between them:
// each CTA brings in 590 KB of weights per layer whatever it does with them.  One buffer has to do then, written when all four CTAs'
// MMAs have read it (a commit that arrives at all of them).  34 to 66 faces, against one launch per layer: 13.7 and 16.1 -> 9.1 us a layer,
// forward of 48 / 64 / 66 faces 544.6 / 595.7 / 608.4 -> 522.2 / 573.1 / 584.9 us.  Four faces a cluster (256 columns, 67 to 132 faces): 16.3 against
// 14.1 and 16.5 us a layer at 80 faces, 17.5 and 20.2 at 128, forward within 1 %; not kept.
//
// A CTA holds, for all channels, its rows and one above and below, in two buffers that take turns.  Its epilogue writes its 128
// channels of its rows into its own next buffer, bytewise, and sends the rows from there by bulk copies: all of them to the CTAs
// with the other channels of the same rows, the first and the last to the CTAs of the neighbouring rows.  What a CTA has made itself is there some 1.5 thousand cycles before the others' bytes, so a layer begins with
// the filter taps that read nothing else: the middle row of taps on its own plane, all nine where the rows are not split.
// (Forward of 1 / 4 / 8 / 15 / 17 / 33 faces, all taps after the last byte -> this: 207 / 222 / 240 / 268 / 311 / 368 -> 201 / 212 / 231 / 259 / 304 / 361 us.)
//
// Bound: latency.  What passes between shared memories goes at 20 B per cycle and CTA whatever instruction sends it (measured:
// 8 KB to 1 / 2 / 4 / 8 CTAs of a cluster of eight 710 / 1110 / 1920 / 3550 cycles by 16-byte st.async, 810 / 1210 / 2005 / 3790 by
// bulk copies), so the split is the one that sends least: at 14x14 16 KB per CTA and layer instead of 36 KB for 2 row tiles x 4
// channel tiles (an earlier kernel with positions as the MMA's rows, the "chain" below).
// Forward of 1 / 4 / 8 / 15 faces, 14x14 stage by that chain -> clusters of eight: 273 / 287 / 309 / 349 -> 230 / 249 / 267 / 304 us; of
// 16 / 17 / 24 / 33 faces, its wide form -> clusters of four: 409 / 413 / 445 / 487 -> 357 / 361 / 396 / 435 us (layers 5.1 -> 3.5 and 7 -> 5 us).
// The 28x28 stage by one launch per layer and the 7x7 one by that chain (from 25 faces a launch per layer): forward of 1 / 8 / 15 /
// 17 / 33 faces 231 / 264 / 302 / 357 / 430 us; with the 28x28 stage here 219 / 250 / 283 / 345 / 408, with the 7x7 one 225 / 262 / 298 / 347 /
// 420, with both 214 / 248 / 279 / 335 / 397.  Their second forms at 1 / 8 / 15 faces: 28x28 223 / 255 / 287, 7x7 219 / 255 / 286.
//
// Replaces, per layer, what conv_tc_kernel does (reference kernels/conv2d_nhwc.c:179-220, kernels/int8_epilogue.c:25-112,
// :253-318); same arithmetic, same bytes.
#include "conv_tc_face.cuh"

namespace {

// C channels on an H x H map, R row tiles; a cluster has C / 128 x R CTAs (rank = row tile * C / 128 + channel tile).  F > 1: a
// cluster takes F faces at once, one under the other with a row of zeros between them, in a single buffer.
template <int C_, int H_, int R_, int F_ = 1>
struct Stage {
    static constexpr int C = C_, H = H_, R = R_, F = F_;
    static constexpr int CT = C / 128;                       // channel tiles = planes of 128 input channels
    static constexpr int CLUSTER = CT * R;
    static constexpr int PITCH = H == 28 ? 32 : H == 14 ? 16 : 8;        // lines of a row: a zero line before it, zero or unread ones behind
    static constexpr int ROW_BYTES = PITCH * 128;
    static constexpr int ROWS = (H + R - 1) / R;             // rows of a tile; where R does not divide H the last tiles have one less
    static constexpr int FACE_ROWS = H + 1;                  // F > 1: rows from a face's first to the next one's
    static constexpr int WIN = F > 1 ? F * FACE_ROWS + 2 : ROWS + 2 + (PITCH == H + 1 ? 1 : 0);      // (a row's last tap may read the line behind it: the next row's zero line)
    static constexpr int BOX_ROWS = F > 1 ? FACE_ROWS : WIN; // rows a face's first input brings
    static constexpr int PARTS = ROWS * PITCH > 256 ? 2 : 1; // of a tile's rows: an MMA has up to 256 columns
    static constexpr int PART_ROWS = ROWS / PARTS;
    static constexpr int PER_GROUP = F > 1 ? (ROWS * F + 3) / 4 : (PART_ROWS + 3) / 4;   // rows of an epilogue group of four warps
    static constexpr int N = F > 1 ? F * FACE_ROWS * PITCH : (ROWS * PITCH + 15) / 16 * 16;
    static constexpr int BUFS = F > 1 ? 1 : 2;
    static constexpr int PLANE_BYTES = WIN * ROW_BYTES;
    static constexpr int ACT_BYTES = CT * PLANE_BYTES;
    // A step of the weight ring: this many planes of one filter tap.  One plane (16 KB) keeps the ring fullest; where four MMAs take
    // 128 cycles or less the issuer does not keep up with that many steps (14x14 with 64 columns: forward of one face 206 -> 215 us).
    // On 7x7 maps with 64 columns and 14x14 with 112, one against two: forward of 16 / 17 / 24 / 33 faces 324 / 325 / 352 / 384 -> 308 / 310 / 337 / 370 us.
    static constexpr int PL_STEP = CT > 1 && N <= (H == 7 ? 32 : 64) ? 2 : 1;
    static constexpr int UNITS = 9 * CT, STEPS = UNITS / PL_STEP;      // a unit: one plane of one tap
    static constexpr int EARLY = R == 1 ? 9 : 3;             // units that read only what this CTA's epilogue has written: they come first
    static constexpr int STEP_BYTES = PL_STEP * 128 * 128;
    static constexpr int OFF_LUT = BUFS * ACT_BYTES;
    static constexpr int OFF_RING = OFF_LUT + FACE_LUT_BYTES;
    static constexpr int FIT = (232448 - 768 - OFF_RING) / STEP_BYTES;
    static constexpr int STAGES = FIT < 12 ? FIT : 12;
    static constexpr int OFF_SH = OFF_RING + STAGES * STEP_BYTES;
    static constexpr uint32_t TMEM_COLS = N <= 32 ? 32 : N <= 64 ? 64 : N <= 128 ? 128 : N <= 256 ? 256 : 512;
    static constexpr int WORDS = (H + 3) / 4;                // a row of a channel in packed bytes
    static constexpr int KEPT_BYTES = H * WORDS * C * 4;     // [row][word][channel]: a warp's 32 channels together
    static_assert(F == 1 || (F == 2 && R == 1 && PITCH == H + 1), "faces of a cluster");
    static_assert(STAGES >= 3 && OFF_RING % 1024 == 0 && ACT_BYTES % 1024 == 0 && N <= 256 * PARTS && ROWS % PARTS == 0, "layout");
    __device__ static int rows(int t) { return H / R + (t < H % R ? 1 : 0); }
    // epilogue group g: its face of the cluster's, its first row in the tile
    __device__ static int group_face(int g) { return F > 1 ? g * F / 4 : 0; }
    __device__ static int group_row(int g) { return F > 1 ? g % (4 / F) * PER_GROUP : g * PER_GROUP; }
    __device__ static int first_row(int t) { return t * (H / R) + (t < H % R ? t : H % R); }
};

struct StageShared {
    uint64_t full[12], empty[12];
    uint64_t a0_full;             // the first input has landed
    uint64_t own_full;            // this CTA's results are in the next layer's input (sixteen warps, each part)
    uint64_t act_full[2];         // the others' are in buffer b's
    uint64_t acc_full;
    uint64_t lut_full, lut_empty;
    uint32_t unit_k[36], unit_db[36];      // of a layer's units in turn: where the weights start, where the activations do (>> 4)
    uint32_t tmem_base;
    int abort_flag;
};

// One layer, or one part of its rows.  RESBN: residual and fused BN (else PReLU); LAST: results go to global memory as NHWC.
template <bool CONTRACT, typename S, bool RESBN, bool LAST>
__device__ __forceinline__ void stage_epilogue(uint8_t* smem, StageShared* sh, const FaceLayer* cl, const float4& k, int L, int rank, int part, int q, int g,
                                               int lane, uint32_t lut_lo, uint32_t lut_hi, int face, int n_faces, int8_t* kept, uint32_t tmem_base,
                                               uint32_t lut_parity, volatile int* abort_flag, const FaceParams& p, bool& ok)
{
    constexpr int PG = S::PER_GROUP, H = S::H, W4 = S::WORDS, CHUNKS = (H + 7) / 8;
    const int h = rank % S::CT, t = rank / S::CT, ch = q * 32 + lane;
    const int n_rows = S::rows(t), r0 = S::first_row(t);
    const int f = S::group_face(g), y0 = part * S::PART_ROWS + S::group_row(g), y1 = S::PARTS > 1 ? (part + 1) * S::PART_ROWS : n_rows;
    const int mine = f >= n_faces ? 0 : y1 - y0 < PG ? y1 - y0 : PG;          // rows of this warp's group: r0 + y0 ..  (may be <= 0)
    const size_t px0 = ((size_t)face * (H * H) + (size_t)(r0 + y0) * H) * S::C + h * 128 + ch;
    kept += (size_t)(part * S::PART_ROWS) * (W4 * S::C * 4);
    uint32_t rw[W4 * PG];
#pragma unroll
    for (int i = 0; i < W4 * PG; i++) rw[i] = 0;
    if (RESBN && ok) {
        const int8_t* res = cl->res;
#pragma unroll
        for (int r = 0; r < PG; r++) {
            if (r >= mine) break;
            if (res) {
#pragma unroll
                for (int c = 0; c < H; c++) {
                    uint32_t b;
                    asm volatile("ld.global.u8 %0, [%1];" : "=r"(b) : "l"(res + px0 + (size_t)(r * H + c) * S::C));
                    rw[W4 * r + c / 4] |= b << (8 * (c & 3));
                }
            } else {
#pragma unroll
                for (int i = 0; i < W4; i++)
                    asm volatile("ld.global.b32 %0, [%1];" : "=r"(rw[W4 * r + i]) : "l"(kept + ((size_t)r * W4 + i) * (S::C * 4)));
            }
        }
    }
    if (RESBN && ok) ok = mbar_wait(smem_u32(&sh->lut_full), lut_parity, abort_flag, p.err, FFCU_ERR_TMA_TIMEOUT, p.wait_cycles);
    if (ok) ok = S::BUFS == 1 ? mbar_wait_cluster(smem_u32(&sh->acc_full), (uint32_t)L & 1, abort_flag, p.err, FFCU_ERR_EPI_TIMEOUT, p.wait_cycles)
                              : mbar_wait(smem_u32(&sh->acc_full), (uint32_t)L & 1, abort_flag, p.err, FFCU_ERR_EPI_TIMEOUT, p.wait_cycles);
    tc_fence_after();
    const uint8_t* lut = smem + S::OFF_LUT;
    const uint32_t taddr = tmem_base + (uint32_t)((f * S::FACE_ROWS + y0) * S::PITCH) + ((uint32_t)(q * 32) << 16);
    const uint32_t s_plane = smem_u32(smem) + (uint32_t)((L + 1) % S::BUFS * S::ACT_BYTES + h * S::PLANE_BYTES);
    const uint32_t s_rows = s_plane + (uint32_t)((f * S::FACE_ROWS + y0 + 1) * S::ROW_BYTES);     // the group's rows in the next input
    if (ok && mine > 0) {
        FaceDst d;
        if (LAST) d.g = cl->out2 + px0;
        else {
#pragma unroll
            for (int i = 0; i < 8; i++) d.ad[i] = (s_rows + (uint32_t)ch) ^ (uint32_t)(i << 4);
        }
        // eight columns at a time, the next ones landing meanwhile
        int va[8], vb[8];
        tmem_ld8_issue(taddr, va);
        TcUnroll<PG * CHUNKS>::run([&](auto uc) {
            constexpr int u = decltype(uc)::value, r = u / CHUNKS, j = u % CHUNKS, n = u + 1;
            constexpr int c0 = 8 * j, c1 = c0 + 8 < H ? c0 + 8 : H;
            int (&v)[8] = u % 2 ? vb : va;
            int (&w)[8] = u % 2 ? va : vb;
            if (r < mine) {
                tmem_ld_wait8(v);
                if (n < PG * CHUNKS && n / CHUNKS < mine) tmem_ld8_issue(taddr + (uint32_t)(n / CHUNKS * S::PITCH + n % CHUNKS * 8), w);
                face_cols<CONTRACT, RESBN, LAST, c0, c1, r, H, S::C, S::PITCH>(v, rw + W4 * r + 2 * j, k, lut, lut_lo, lut_hi, d);
            }
        });
    }
    if (!LAST) {
        // Every warp comes here whatever its ok flag: none may be left waiting.  (What the warps have read of the accumulator
        // counts with the same arrival.)
        fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && ok) mbar_arrive(smem_u32(&sh->own_full));
        asm volatile("bar.sync %0, 128;" ::"r"(2 + g) : "memory");
        if (ok && mine > 0) {
            const uint32_t bar = smem_u32(&sh->act_full[(L + 1) % S::BUFS]);
            const uint32_t tile0 = (uint32_t)(t * S::CT);                  // rank of this row tile's first CTA
            if (q == 0) {
                // all rows: to the CTAs with the tile's other channels
                if (lane < S::CT - 1) {
                    const uint32_t to = tile0 + (uint32_t)((h + 1 + lane) % S::CT);
                    bulk_send(map_to_cta(s_rows, to), s_rows, (uint32_t)(mine * S::ROW_BYTES), map_to_cta(bar, to));
                }
            } else if (q == 1) {
                // the first row is the row below the tile above's
                if (y0 == 0 && t > 0 && lane < S::CT) {
                    const uint32_t to = tile0 - (uint32_t)(S::CT - lane);
                    bulk_send(map_to_cta(s_plane + (uint32_t)((S::rows(t - 1) + 1) * S::ROW_BYTES), to), s_rows, S::ROW_BYTES, map_to_cta(bar, to));
                }
            } else if (q == 2) {
                // the last one the row above the tile below's
                if (y0 + mine == n_rows && t < S::R - 1 && lane < S::CT) {
                    const uint32_t to = tile0 + (uint32_t)(S::CT + lane);
                    bulk_send(map_to_cta(s_plane, to), s_plane + (uint32_t)(n_rows * S::ROW_BYTES), S::ROW_BYTES, map_to_cta(bar, to));
                }
            }
        }
    }
    if (ok && RESBN && !LAST) {
#pragma unroll
        for (int i = 0; i < PG * W4; i++)
            if (i / W4 < mine) asm volatile("st.global.b32 [%0], %1;" ::"l"(kept + (size_t)i * (S::C * 4)), "r"(rw[i]) : "memory");
    }
    if (ok && LAST) {
        int8_t* out = cl->out + px0;
#pragma unroll
        for (int r = 0; r < PG; r++)
            if (r < mine) {
#pragma unroll
                for (int c = 0; c < H; c++) out[(r * H + c) * S::C] = (int8_t)(rw[W4 * r + c / 4] >> (8 * (c & 3)));
            }
    }
}

template <bool CONTRACT, typename S>
__global__ void __launch_bounds__(TC_THREADS, 1)
conv_stage_kernel(const __grid_constant__ CUtensorMap mapA, const FaceParams p)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    StageShared* sh = (StageShared*)(smem + S::OFF_SH);
    if (smem_u32(smem) & 1023) {                              // the swizzle atoms' alignment, as the declaration asks for it
        if (threadIdx.x == 0) atomicCAS(p.err, 0, FFCU_ERR_TMA_TIMEOUT);
        return;
    }
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int rank = (int)cluster_ctarank();
    const int cluster = (int)blockIdx.x / S::CLUSTER, n_faces = p.faces - cluster * S::F < S::F ? p.faces - cluster * S::F : S::F;
    const int h = rank % S::CT, t = rank / S::CT;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S::STAGES; s++) { mbar_init(smem_u32(&sh->full[s]), 1); mbar_init(smem_u32(&sh->empty[s]), 1); }
        mbar_init(smem_u32(&sh->a0_full), 1);
        mbar_init(smem_u32(&sh->own_full), 16 * S::PARTS);
        for (int b = 0; b < 2; b++) mbar_init(smem_u32(&sh->act_full[b]), 1);          // the arming arrival
        mbar_init(smem_u32(&sh->acc_full), S::BUFS == 1 ? S::CLUSTER : 1);              // one buffer: nobody reads it any more
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
    if (threadIdx.x >= 32 && threadIdx.x < 32 + S::UNITS) {
        // own plane first, of that the middle row of taps
        const int u = (int)threadIdx.x - 32, t9 = u % 9, plane = (h + u / 9) % S::CT;
        const int kh = u >= 9 || S::R == 1 ? t9 / 3 : t9 < 3 ? 1 : t9 < 6 ? 0 : 2, kw = t9 % 3;
        sh->unit_k[u] = (uint32_t)(((kh * 3 + kw) * S::CT + plane) * 128);
        sh->unit_db[u] = (uint32_t)((kh * S::ROW_BYTES + kw * 128 + plane * S::PLANE_BYTES) >> 4);
    }
    if (S::BUFS == 2) {
        // The second buffer's padding.  By stores in front of the cluster's barrier, not by a load of the first input as in the first buffer: the
        // peers wait for their own loads only, and their first layer's rows may be here before a load of this CTA's has landed.
        for (int i = threadIdx.x; i < S::ACT_BYTES / 16; i += TC_THREADS) *(int4*)(smem + S::ACT_BYTES + i * 16) = make_int4(0, 0, 0, 0);
        fence_async_smem();
    }
    if (S::F > 1) {
        // the two rows below the last face (the others' zeros come with the first input)
        for (int i = threadIdx.x; i < S::CT * 2 * S::ROW_BYTES / 16; i += TC_THREADS)
            *(int4*)(smem + i / (2 * S::ROW_BYTES / 16) * S::PLANE_BYTES + S::F * S::FACE_ROWS * S::ROW_BYTES + i % (2 * S::ROW_BYTES / 16) * 16) = make_int4(0, 0, 0, 0);
        fence_async_smem();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                       // the peers' barriers are initialised
    tc_fence_after();
    const uint32_t tmem_base = sh->tmem_base;
    volatile int* abort_flag = &sh->abort_flag;
    const uint32_t s0 = smem_u32(smem);

    if (warp == TC_PRODUCER_WARP) {
        // Weight producer: a unit is a box (lane i: the step's unit i)
        int stage = 0, gs = 0; uint32_t phase = 0;
        bool ok = true;
#pragma unroll 1
        for (int L = 0; L < p.n_layers && ok; L++) {
            const CUtensorMap* map = &p.layers[L].mapB;
            if (lane < S::PL_STEP) asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
#pragma unroll 1
            for (int st = 0; st < S::STEPS; st++, gs++) {
                ok = mbar_wait(smem_u32(&sh->empty[stage]), phase ^ 1, abort_flag, p.err, FFCU_ERR_EMPTY_TIMEOUT, p.wait_cycles);
                if (!ok) break;
                if (lane == 0) mbar_expect_tx(smem_u32(&sh->full[stage]), S::STEP_BYTES);
                __syncwarp();
                // (drop_step: the timeout test's launch, CTA 0 leaves out this step)
                if (lane < S::PL_STEP && (gs != p.drop_step || rank != 0))
                    tma_load_4d(s0 + S::OFF_RING + stage * S::STEP_BYTES + lane * (128 * 128), map, smem_u32(&sh->full[stage]),
                                (int)sh->unit_k[st * S::PL_STEP + lane], h * 128, 0, 0);
                if (++stage == S::STAGES) { stage = 0; phase ^= 1; }
            }
        }
    } else if (warp == TC_ISSUER_WARP) {
        if (tc_elect_one()) {
            constexpr uint32_t IDESC = idesc_i8(S::N / S::PARTS);
            const uint32_t full0 = smem_u32(&sh->full[0]), empty0 = smem_u32(&sh->empty[0]);
            const uint64_t da0 = smem_desc<128>(s0 + S::OFF_RING);
            // what this CTA receives of each layer: its rows' other channels, and the rows above and below
            const uint32_t in_bytes = (uint32_t)(S::ROW_BYTES * ((S::CT - 1) * S::rows(t) * n_faces + S::CT * ((t > 0) + (t < S::R - 1))));
            int stage = 0; uint32_t phase = 0, ready = 0;
            bool ok = true;
#pragma unroll 1
            for (int L = 0; L < p.n_layers && ok; L++) {
                const int buf = L % S::BUFS;
                // (bytes that land before this only drive the count negative: the phase needs this arrival)
                if (S::BUFS == 2 && L + 1 < p.n_layers) mbar_expect_tx(smem_u32(&sh->act_full[buf ^ 1]), in_bytes);
                ok = L == 0 ? mbar_wait(smem_u32(&sh->a0_full), 0, abort_flag, p.err, FFCU_ERR_TMA_TIMEOUT, p.wait_cycles)
                            : mbar_wait(smem_u32(&sh->own_full), (uint32_t)(L - 1) & 1, abort_flag, p.err, FFCU_ERR_TMA_TIMEOUT, p.wait_cycles);
                if (!ok) break;
                tc_fence_after();
                const uint64_t db0 = smem_desc<128>(s0 + (uint32_t)(buf * S::ACT_BYTES));
#pragma unroll 1
                for (int u = 0; u < S::UNITS && ok;) {
                    if (!ready) {
                        ok = mbar_wait(full0 + stage * 8, phase, abort_flag, p.err, FFCU_ERR_TMA_TIMEOUT, p.wait_cycles);
                        if (!ok) break;
                    }
                    int ns = stage + 1; uint32_t np = phase;
                    if (ns == S::STAGES) { ns = 0; np ^= 1; }
                    ready = mbar_test(full0 + ns * 8, np);                       // used next round
                    tc_fence_after();
                    const uint64_t da = da0 + (uint64_t)((uint32_t)(stage * S::STEP_BYTES) >> 4);
#pragma unroll
                    for (int pl = 0; pl < S::PL_STEP; pl++, u++) {
                        if (u == S::EARLY) {
                            if (L) ok = mbar_wait_cluster(smem_u32(&sh->act_full[buf]), (uint32_t)((L - 1) / S::BUFS) & 1, abort_flag, p.err, FFCU_ERR_TMA_TIMEOUT, p.wait_cycles);
                            if (!ok) break;
                            if (S::BUFS == 1 && L + 1 < p.n_layers) mbar_expect_tx(smem_u32(&sh->act_full[0]), in_bytes);
                            tc_fence_after();
                        }
                        const uint64_t db = db0 + sh->unit_db[u];
#pragma unroll
                        for (int part = 0; part < S::PARTS; part++)
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                umma_i8(tmem_base + (uint32_t)(part * (S::N / S::PARTS)), da + (uint64_t)(pl * (128 * 128 >> 4) + 2 * k),
                                        db + (uint64_t)((part * S::PART_ROWS * S::ROW_BYTES >> 4) + 2 * k), IDESC, (u | k) ? 1u : 0u);
                    }
                    if (!ok) break;
                    umma_commit(empty0 + stage * 8);
                    stage = ns; phase = np;
                }
                if (!ok) break;
                if (S::BUFS == 1) umma_commit_multicast(smem_u32(&sh->acc_full), (uint16_t)((1 << S::CLUSTER) - 1));
                else umma_commit(smem_u32(&sh->acc_full));
            }
        }
    } else if (warp == TC_ISSUER2_WARP) {
        // The face's first input, and the fused BNs' byte tables
        if (tc_elect_one()) {
            tc_pdl_wait();
            const long long hold = rank == 0 ? p.hold_cycles : 0;
            tc_hold(hold);
            mbar_expect_tx(smem_u32(&sh->a0_full), S::F * S::CT * S::BOX_ROWS * S::ROW_BYTES);
#pragma unroll
            for (int i = 0; i < S::F * S::CT; i++)
                tma_load_4d(s0 + i % S::CT * S::PLANE_BYTES + i / S::CT * (S::FACE_ROWS * S::ROW_BYTES), &mapA, smem_u32(&sh->a0_full),
                            i % S::CT * 128, -1, S::first_row(t) - 1, p.face0 + cluster * S::F + i / S::CT);
            uint32_t lut_par = 0;
            bool ok = true;
#pragma unroll 1
            for (int L = 0; L < p.n_layers && ok; L++) {
                const uint8_t* lut = p.layers[L].lut;
                if (!lut) continue;
                // (twice the limit: whoever this wait depends on gives up first, and says where)
                ok = mbar_wait(smem_u32(&sh->lut_empty), lut_par ^ 1, abort_flag, p.err, FFCU_ERR_EMPTY_TIMEOUT, 2 * p.wait_cycles);
                lut_par ^= 1;
                if (!ok) break;
                mbar_expect_tx(smem_u32(&sh->lut_full), FACE_LUT_BYTES);
                bulk_load(s0 + S::OFF_LUT, lut + h * FACE_LUT_BYTES, FACE_LUT_BYTES, smem_u32(&sh->lut_full));
                tc_hold(hold);
            }
        }
    } else {
        const int q = warp & 3, g = warp >> 2;
        const uint32_t lut_lo = (uint32_t)(lane * 4 + (q & 1) * 128) * 0x01010101u, lut_hi = (uint32_t)(q >> 1) * 0x01010101u;
        // a result that the next residual layer adds lies as its thread left it
        const int slot = cluster * S::F + S::group_face(g), face = p.face0 + slot;
        int8_t* kept = p.kept + (size_t)slot * S::KEPT_BYTES + ((size_t)(S::first_row(t) + S::group_row(g)) * S::WORDS * S::C + h * 128 + q * 32 + lane) * 4;      // (its first part's)
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
#pragma unroll 1
            for (int part = 0; part < S::PARTS; part++) {
                if (last)    stage_epilogue<CONTRACT, S, true, true>(smem, sh, cl, k, L, rank, part, q, g, lane, lut_lo, lut_hi, face, n_faces, kept, tmem_base, lut_par, abort_flag, p, ok);
                else if (bn) stage_epilogue<CONTRACT, S, true, false>(smem, sh, cl, k, L, rank, part, q, g, lane, lut_lo, lut_hi, face, n_faces, kept, tmem_base, lut_par, abort_flag, p, ok);
                else         stage_epilogue<CONTRACT, S, false, false>(smem, sh, cl, k, L, rank, part, q, g, lane, lut_lo, lut_hi, face, n_faces, kept, tmem_base, lut_par, abort_flag, p, ok);
            }
            if (bn) {
                lut_par ^= 1;
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sh->lut_empty));
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

static_assert(sizeof(StageShared) <= 768, "StageShared: what the ring leaves");
template <typename S>
constexpr int smem_bytes() { return S::OFF_SH + (int)sizeof(StageShared); }

template <bool CONTRACT, typename S>
int set_smem()
{
    static int done[64] = {};             // per device: the attribute belongs to the device's copy of the function
    int dev = 0;
    FFCU_CHECK(cudaGetDevice(&dev));
    if (!done[dev & 63]) {
        FFCU_CHECK(cudaFuncSetAttribute(conv_stage_kernel<CONTRACT, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<S>()));
        done[dev & 63] = 1;
    }
    return 0;
}

template <typename S>
int launch(int mode, int faces, cudaStream_t s, const CUtensorMap& mapA, const FaceParams& prm)
{
    const int rc = mode ? set_smem<true, S>() : set_smem<false, S>();
    if (rc != 0) return rc;
    return mode ? tc_launch_ex(conv_stage_kernel<true, S>, S::CLUSTER * ((faces + S::F - 1) / S::F), smem_bytes<S>(), s, S::CLUSTER, mapA, prm)
                : tc_launch_ex(conv_stage_kernel<false, S>, S::CLUSTER * ((faces + S::F - 1) / S::F), smem_bytes<S>(), s, S::CLUSTER, mapA, prm);
}

template <typename S>
StageForm form()
{
    StageForm f = {S::BOX_ROWS, S::PITCH, S::KEPT_BYTES * S::F, 0, S::F};
    if (set_smem<true, S>() != 0 || set_smem<false, S>() != 0) { cudaGetLastError(); return f; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(S::CLUSTER);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smem_bytes<S>();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S::CLUSTER; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, conv_stage_kernel<true, S>, &cfg) != cudaSuccess) { cudaGetLastError(); return f; }
    f.clusters = n;
    return f;
}

// calls fn with the form of the stage of H x H maps: 0, more and smaller tiles (few faces), 1, or 2 (not 14x14; 7x7: two
// faces a cluster)
template <typename Fn>
auto with_form(int H, int i, Fn&& fn)
{
    if (H == 28) return i == 0 ? fn(Stage<128, 28, 7>{}) : i == 1 ? fn(Stage<128, 28, 4>{}) : fn(Stage<128, 28, 2>{});
    if (H == 7) return i == 0 ? fn(Stage<512, 7, 2>{}) : i == 1 ? fn(Stage<512, 7, 1>{}) : fn(Stage<512, 7, 1, 2>{});
    return i == 0 ? fn(Stage<256, 14, 4>{}) : fn(Stage<256, 14, 2>{});
}

}  // namespace

StageForm tc_stage_form(int H, int i) { return with_form(H, i, [](auto s) { return form<decltype(s)>(); }); }

int tc_launch_stage(int H, int i, int mode, int faces, cudaStream_t s, const CUtensorMap& mapA, const FaceParams& prm)
{
    return with_form(H, i, [&](auto st) { return launch<decltype(st)>(mode, faces, s, mapA, prm); });
}
