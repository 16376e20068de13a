// conv_tc_face.cu -- the 14x14 stage (a run of 3x3 stride-1 256 -> 256 convolutions) in ONE launch, a CTA pair per
// face, with the activations resident in shared memory through all layers.
//
// The operands change places against the other kernels: the weights are the MMA's 256 rows (128 output channels per CTA
// of the pair) and the face's positions its columns.  So
//   * a face is 14 rows of 16 lines = 224 columns (12.5 % of them padding; as rows of 128 positions it would be 256),
//   * an epilogue thread owns one output channel: its constants sit in registers, and only positions that exist are walked,
//   * the fused BN's byte table is laid out so that a warp's 32 look-ups, one per channel, fall into 32 banks.
// Each CTA holds 7 of the image's rows and one above and below (9 x 16 lines of 128 B per 128-channel plane, as a TMA load
// with 128-byte swizzle leaves them), so filter tap (kh, kw) is the same buffer read kh * 16 + kw lines further on.  A layer's
// result is written over its input: by the time the accumulator is complete no MMA reads that any more.  The half that
// belongs to the other CTA's rows goes through a staging buffer and one bulk copy of 4 KB per 32-channel-group of warps.
// Weights stream through a TMA ring that runs ahead across layers.  Two faces take turns in a pair, so that one's MMAs
// cover the other's epilogue and exchange; a face left over runs alone.
//
// Bound: the tensor pipe with two faces per pair (86 % active; a face and layer take 9.2 thousand cycles, 72 MMAs of 112 are
// 8.1), latency with one: 13-15 thousand cycles, of which the MMAs 8.9, the epilogue 3.1 (PReLU) or 4.6 (residual + BN; the
// half-rate integer pipe and the look-ups), the exchange 1.5.  Forward of 34 / 64 / 74 / 75 / 100 / 148 / 256 / 512 / 1024 faces, one
// launch per layer -> this: 560 / 744 / 771 / 776 / 1002 / 1240 / 1925 / 3500 / 6800 -> 491 / 613 / 636 / 698 / 805 / 1007 / 1750 / 3150 /
// 6420 us.  Up to the 33 faces or so that the device holds clusters of four for, those are quicker (conv_tc_stage.cu).
// Tried and not kept: one warp that sends all staging buffers (its five copies one after another: +14 us at 64 faces), one remote
// arrival per CTA behind local ones (+9 us), the epilogue as a loop over rows or pairs of rows (loads' latency, spills: +20-30 us).
//
// Replaces, per layer, what conv_tc2_kernel does (reference kernels/conv2d_nhwc.c:179-220, kernels/int8_epilogue.c:25-112,
// :253-318); same arithmetic, same bytes.
#include "conv_tc_face.cuh"

namespace {

constexpr int STEP_BYTES = 128 * 128;                        // one tap of one plane: 128 output channels x 128 input channels
constexpr int PLANE_BYTES = 9 * 16 * 128;
constexpr int ACT_BYTES = 2 * PLANE_BYTES;
constexpr int STG_BYTES = 8 * 16 * 128;                      // the eight rows the other CTA reads
constexpr int LUT_BYTES = FACE_LUT_BYTES;
constexpr int STEPS = 18;                                    // per layer: nine taps of two planes
constexpr int OFF_STG = 2 * ACT_BYTES;
constexpr int OFF_LUT = OFF_STG + 2 * STG_BYTES;
constexpr int OFF_RING = OFF_LUT + LUT_BYTES;
constexpr int OFF_SH = OFF_RING + FACE_STAGES * STEP_BYTES;
static_assert(OFF_STG % 1024 == 0 && OFF_RING % 1024 == 0, "swizzle atoms");

struct FaceShared {
    uint64_t full[FACE_STAGES];
    uint64_t empty[FACE_STAGES];
    uint64_t a0_full[2];          // (leader) slot's first input has landed in both CTAs
    uint64_t acc_full[2];         // slot's accumulator is complete
    uint64_t in_ready[2];         // (leader) both CTAs' own results are in place, and what came to CTA 1 from its peer
    uint64_t rx[2];               // what comes to this CTA from its peer has landed
    uint64_t face_done[2];        // slot's last layer: its MMAs are done (for those who do not follow acc_full through all layers)
    uint64_t lut_full, lut_empty;
    uint32_t tmem_base;
    int abort_flag;
};

// One thread of the epilogue: its channel and its warp's share of the rows.  Warps are (TMEM lane quarter q, group g); a
// group takes two of the eight rows the other CTA reads, first, and three half rows of the six that only this CTA reads.
struct FaceEpi {
    int rank, g, q, lane, ch;     // ch: channel within the CTA's 128
    int row_tx, hr_own;           // first row of the former, first half row of the latter
    uint32_t lut_lo, lut_hi;
    uint32_t peer;
};

// One layer of one face.  RESBN: residual and fused BN (else PReLU); LAST: results go to global memory as NHWC.
template <bool CONTRACT, bool RESBN, bool LAST>
__device__ __forceinline__ void face_epilogue(uint8_t* smem, FaceShared* sh, const FaceEpi& e, const FaceLayer* cl, const float4& k,
                                              int slot, int face, uint32_t tmem_base, uint32_t acc_parity, uint32_t leader_ready,
                                              bool wait_lut, uint32_t lut_parity, volatile int* abort_flag, const FaceParams& p, bool& ok)
{
    uint32_t rw[14];
#pragma unroll
    for (int i = 0; i < 14; i++) rw[i] = 0;
    const size_t px0 = (size_t)face * 196 * FACE_C + e.rank * 128 + e.ch;          // NHWC: first pixel's byte of this channel
    auto half_row = [&](int i) { return i < 4 ? 2 * e.row_tx + i : e.hr_own + i - 4; };
    // a result that the next residual layer adds lies as its thread left it: eight positions of a channel together
    int8_t* kept = p.kept + (size_t)((blockIdx.x >> 1) * 2 + slot) * FACE_KEPT_BYTES + (e.rank * 128 + e.ch) * 8;
    if (RESBN && ok) {
        const int8_t* res = cl->res;
        if (res) {
#pragma unroll
            for (int i = 0; i < 7; i++) {
                const int hr = half_row(i), n = hr & 1 ? 6 : 8;
                const int8_t* s = res + px0 + (size_t)((hr >> 1) * 14 + (hr & 1) * 8) * FACE_C;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    uint32_t b = 0;
                    if (j < n) asm volatile("ld.global.u8 %0, [%1];" : "=r"(b) : "l"(s + j * FACE_C));
                    rw[2 * i + j / 4] |= b << (8 * (j & 3));
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < 7; i++)
                asm volatile("ld.global.v2.b32 {%0, %1}, [%2];" : "=r"(rw[2 * i]), "=r"(rw[2 * i + 1]) : "l"(kept + half_row(i) * (FACE_C * 8)));
        }
    }
    if (ok && wait_lut) ok = mbar_wait(smem_u32(&sh->lut_full), lut_parity, abort_flag, p.err, FFCU_ERR_TMA_TIMEOUT, p.wait_cycles);
    if (ok) ok = mbar_wait(smem_u32(&sh->acc_full[slot]), acc_parity, abort_flag, p.err, FFCU_ERR_EPI_TIMEOUT, p.wait_cycles);
    tc_fence_after();
    const uint8_t* lut = smem + OFF_LUT;
    const uint32_t taddr = tmem_base + (uint32_t)(slot * 256) + ((uint32_t)(e.q * 32) << 16);
    const uint32_t s_act = smem_u32(smem) + (uint32_t)(slot * ACT_BYTES + e.rank * PLANE_BYTES);
    const uint32_t s_stg = smem_u32(smem) + (uint32_t)(OFF_STG + slot * STG_BYTES + e.g * 4096);
    const uint32_t byte0 = (uint32_t)((e.ch >> 4) << 4 | (e.ch & 15));
    FaceDst d;
    auto aim = [&](uint32_t base) {
#pragma unroll
        for (int i = 0; i < 8; i++) d.ad[i] = (base + byte0) ^ (uint32_t)(i << 4);
    };
    // Half a row at a time, the next one's accumulators landing meanwhile (whole rows: 16 registers more, and spills).
    int v0[8], v1[8];
    auto fetch = [&](int i, int (&v)[8]) { tmem_ld8_issue(taddr + (uint32_t)(half_row(i) * 8), v); };
    if (ok) {
        fetch(0, v0);
        if (LAST) d.g = cl->out2 + px0 + (size_t)(e.row_tx * 14) * FACE_C;
        else aim(s_stg);
        tmem_ld_wait8(v0);
        fetch(1, v1);
        face_half_a<CONTRACT, RESBN, LAST, 0>(v0, rw + 0, k, lut, e.lut_lo, e.lut_hi, d);
        tmem_ld_wait8(v1);
        fetch(2, v0);
        face_half_b<CONTRACT, RESBN, LAST, 0>(v1, rw + 2, k, lut, e.lut_lo, e.lut_hi, d);
        tmem_ld_wait8(v0);
        fetch(3, v1);
        face_half_a<CONTRACT, RESBN, LAST, 1>(v0, rw + 4, k, lut, e.lut_lo, e.lut_hi, d);
        tmem_ld_wait8(v1);
        fetch(4, v0);
        face_half_b<CONTRACT, RESBN, LAST, 1>(v1, rw + 6, k, lut, e.lut_lo, e.lut_hi, d);
    }
    if (!LAST) {
        // the group's two rows are 4 KB that lie alike here and there (the padding's zeros included).  Every warp comes here
        // whatever its ok flag: none may be left waiting.
        fence_async_smem();
        asm volatile("bar.sync %0, 128;" ::"r"(2 + e.g) : "memory");
        if (ok) {
            if (e.q == 0 && e.lane == 0)
                bulk_send(map_to_cta(s_act + (uint32_t)(e.rank * 2048 + e.g * 4096), e.peer), s_stg, 4096, map_to_cta(smem_u32(&sh->rx[slot]), e.peer));
            if (e.g == (e.rank ? 3 : 0)) {
                // rows 6 and 7 are read by both CTAs
                const uint32_t t = (uint32_t)((e.q * 32 + e.lane) * 16), dst = s_act + (e.rank ? 0u : 7u * 2048u) + t;
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    int x, y, z, w;
                    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(x), "=r"(y), "=r"(z), "=r"(w) : "r"(s_stg + t + i * 2048));
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + i * 2048), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
                }
            }
        }
    }
    if (ok) {
        const int row = e.hr_own >> 1;
        if (LAST) d.g = cl->out2 + px0 + (size_t)(row * 14) * FACE_C;
        else aim(s_act + (uint32_t)((e.rank ? row - 6 : row + 1) * 2048));
        tmem_ld_wait8(v0);
        fetch(5, v1);
        if (e.g & 1) {
            face_half_b<CONTRACT, RESBN, LAST, 0>(v0, rw + 8, k, lut, e.lut_lo, e.lut_hi, d);
            tmem_ld_wait8(v1);
            fetch(6, v0);
            face_half_a<CONTRACT, RESBN, LAST, 1>(v1, rw + 10, k, lut, e.lut_lo, e.lut_hi, d);
            tmem_ld_wait8(v0);
            face_half_b<CONTRACT, RESBN, LAST, 1>(v0, rw + 12, k, lut, e.lut_lo, e.lut_hi, d);
        } else {
            face_half_a<CONTRACT, RESBN, LAST, 0>(v0, rw + 8, k, lut, e.lut_lo, e.lut_hi, d);
            tmem_ld_wait8(v1);
            fetch(6, v0);
            face_half_b<CONTRACT, RESBN, LAST, 0>(v1, rw + 10, k, lut, e.lut_lo, e.lut_hi, d);
            tmem_ld_wait8(v0);
            face_half_a<CONTRACT, RESBN, LAST, 1>(v0, rw + 12, k, lut, e.lut_lo, e.lut_hi, d);
        }
    }
    if (!LAST) fence_async_smem();
    tc_fence_before();
    __syncwarp();
    // (the global stores come after it: a release waits for what the warp has stored before)
    if (e.lane == 0 && ok) mbar_arrive_release_cluster(leader_ready + (uint32_t)(slot * 8));
    if (ok && RESBN && !LAST) {
#pragma unroll
        for (int i = 0; i < 7; i++)
            asm volatile("st.global.v2.b32 [%0], {%1, %2};" ::"l"(kept + half_row(i) * (FACE_C * 8)), "r"(rw[2 * i]), "r"(rw[2 * i + 1]) : "memory");
    }
    if (ok && LAST) {
        int8_t* out = cl->out + px0;
#pragma unroll
        for (int i = 0; i < 7; i++) {
            const int hr = half_row(i), n = hr & 1 ? 6 : 8;
            int8_t* o = out + (size_t)((hr >> 1) * 14 + (hr & 1) * 8) * FACE_C;
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (j < n) o[j * FACE_C] = (int8_t)(rw[2 * i + j / 4] >> (8 * (j & 3)));
        }
    }
}

template <bool CONTRACT>
__global__ void __launch_bounds__(TC_THREADS, 1)
conv_face_kernel(const __grid_constant__ CUtensorMap mapA, const FaceParams p)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    FaceShared* sh = (FaceShared*)(smem + OFF_SH);
    if (smem_u32(smem) & 1023) {                              // the swizzle atoms' alignment, as the declaration asks for it
        if (threadIdx.x == 0) atomicCAS(p.err, 0, FFCU_ERR_TMA_TIMEOUT);
        return;
    }
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();                  // 0 = leader
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int nf = (p.faces - pair + n_pairs - 1) / n_pairs;  // this pair's faces: pair, pair + n_pairs, ...
    const int rounds = (nf + 1) >> 1;                         // two at a time, slots 0 and 1

    if (threadIdx.x == 0) {
        for (int s = 0; s < FACE_STAGES; s++) { mbar_init(smem_u32(&sh->full[s]), 1); mbar_init(smem_u32(&sh->empty[s]), 1); }
        for (int s = 0; s < 2; s++) {
            mbar_init(smem_u32(&sh->a0_full[s]), 1);
            mbar_init(smem_u32(&sh->acc_full[s]), 1);
            mbar_init(smem_u32(&sh->in_ready[s]), 33);        // both CTAs' epilogue warps, CTA 1's word that its rx is complete
            mbar_init(smem_u32(&sh->rx[s]), 1);
            mbar_init(smem_u32(&sh->face_done[s]), 1);
        }
        mbar_init(smem_u32(&sh->lut_full), 1);
        mbar_init(smem_u32(&sh->lut_empty), 16);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < 2 * STG_BYTES / 16; i += TC_THREADS)      // the padding's lines stay zero
        *(int4*)(smem + OFF_STG + i * 16) = make_int4(0, 0, 0, 0);
    fence_async_smem();
    if (warp == TC_ISSUER_WARP) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&sh->tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                       // the peer's barriers are initialised
    tc_fence_after();
    const uint32_t tmem_base = sh->tmem_base;
    volatile int* abort_flag = &sh->abort_flag;
    const uint32_t s0 = smem_u32(smem);

    if (warp == TC_PRODUCER_WARP) {
        // Weight producer: every layer's 18 steps, once per face; each CTA fetches its 128 output channels' half, counted on
        // the leader's barrier.
        const uint32_t full_leader = map_to_cta(smem_u32(&sh->full[0]), 0);
        int stage = 0, gs = 0; uint32_t phase = 0;
        bool ok = true;
#pragma unroll 1
        for (int i = 0; i < rounds && ok; i++) {
            const int slots = nf - 2 * i < 2 ? 1 : 2;
#pragma unroll 1
            for (int L = 0; L < p.n_layers && ok; L++) {
                const CUtensorMap* map = &p.layers[L].mapB;
                if (lane == 0) asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
#pragma unroll 1
                for (int st = 0, x = 0; st < STEPS * slots; st++, gs++) {
                    ok = mbar_wait(smem_u32(&sh->empty[stage]), phase ^ 1, abort_flag, p.err, FFCU_ERR_EMPTY_TIMEOUT, p.wait_cycles);
                    if (!ok) break;
                    if (lane == 0) {
                        if (rank == 0) mbar_expect_tx(smem_u32(&sh->full[stage]), 2 * STEP_BYTES);
                        // (drop_step: the timeout test's launch, CTA 0 leaves out this step)
                        if (gs != p.drop_step || rank != 0)
                            tma2_load_4d(s0 + OFF_RING + stage * STEP_BYTES, map, full_leader + stage * 8, x, (int)rank * 128, 0, 0);
                    }
                    __syncwarp();
                    if (++stage == FACE_STAGES) { stage = 0; phase ^= 1; }
                    x += 128;
                    if (x == STEPS * 128) x = 0;
                }
            }
        }
    } else if (warp == TC_ISSUER_WARP && rank == 0) {
        if (tc_elect_one()) {
            // MMA issuer (leader CTA)
            constexpr uint32_t IDESC = idesc_i8(224, 256);
            const uint32_t full0 = smem_u32(&sh->full[0]), empty0 = smem_u32(&sh->empty[0]);
            const uint64_t da0 = smem_desc<128>(s0 + OFF_RING);
            int stage = 0; uint32_t phase = 0, ready = 0;
            uint32_t in_par = 0, rx_par = 0;                  // bit s: slot s
            bool ok = true;
#pragma unroll 1
            for (int i = 0; i < rounds && ok; i++) {
                const int slots = nf - 2 * i < 2 ? 1 : 2;
#pragma unroll 1
                for (int L = 0; L < p.n_layers && ok; L++) {
#pragma unroll 1
                    for (int s = 0; s < slots && ok; s++) {
                        const uint32_t bit = 1u << s;
                        if (L == 0) ok = mbar_wait(smem_u32(&sh->a0_full[s]), (uint32_t)i & 1, abort_flag, p.err, FFCU_ERR_TMA_TIMEOUT, p.wait_cycles);
                        else {
                            ok = mbar_wait_cluster(smem_u32(&sh->rx[s]), (rx_par >> s) & 1, abort_flag, p.err, FFCU_ERR_TMA_TIMEOUT, p.wait_cycles);
                            rx_par ^= bit;
                        }
                        if (ok && (L | i)) {                  // (first layer: the previous face's accumulator has been read)
                            ok = mbar_wait_cluster(smem_u32(&sh->in_ready[s]), (in_par >> s) & 1, abort_flag, p.err, FFCU_ERR_TMEM_TIMEOUT, p.wait_cycles);
                            in_par ^= bit;
                        }
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t d_tmem = tmem_base + (uint32_t)(s * 256);
                        uint64_t db_row = smem_desc<128>(s0 + (uint32_t)(s * ACT_BYTES));
                        uint32_t first = 0;
#pragma unroll 1
                        for (int kh = 0; kh < 3 && ok; kh++, db_row += 16 * 128 / 16) {
#pragma unroll
                            for (int kp = 0; kp < 6; kp++) {  // (kw, plane)
                                if (!ready) {
                                    ok = mbar_wait_cluster(full0 + stage * 8, phase, abort_flag, p.err, FFCU_ERR_TMA_TIMEOUT, p.wait_cycles);
                                    if (!ok) break;
                                }
                                int ns = stage + 1; uint32_t np = phase;
                                if (ns == FACE_STAGES) { ns = 0; np ^= 1; }
                                ready = mbar_test_cluster(full0 + ns * 8, np);       // used next round
                                tc_fence_after();
                                const uint64_t da = da0 + (uint64_t)((uint32_t)(stage * STEP_BYTES) >> 4);
                                const uint64_t db = db_row + (uint64_t)(((kp >> 1) * 128 + (kp & 1) * PLANE_BYTES) >> 4);
#pragma unroll
                                for (int k = 0; k < 4; k++)
                                    umma2_i8(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), IDESC, (kp | k) ? 1u : first);
                                first = 1;
                                umma2_commit_both(empty0 + stage * 8);
                                stage = ns; phase = np;
                            }
                        }
                        if (!ok) break;
                        umma2_commit_both(smem_u32(&sh->acc_full[s]));
                        // arm the barrier of what will come from the peer (bytes that land before this would only drive the
                        // count negative: the phase needs this arrival)
                        if (L + 1 < p.n_layers) mbar_expect_tx(smem_u32(&sh->rx[s]), STG_BYTES);
                        else umma2_commit_both(smem_u32(&sh->face_done[s]));
                    }
                }
            }
        }
    } else if (warp == TC_ISSUER_WARP) {
        if (tc_elect_one()) {
            // CTA 1: tells the leader when what comes from it has landed
            const uint32_t leader_ready = map_to_cta(smem_u32(&sh->in_ready[0]), 0);
            uint32_t rx_par = 0;
            bool ok = true;
#pragma unroll 1
            for (int i = 0; i < rounds && ok; i++) {
                const int slots = nf - 2 * i < 2 ? 1 : 2;
#pragma unroll 1
                for (int L = 0; L < p.n_layers && ok; L++) {
#pragma unroll 1
                    for (int s = 0; s < slots && ok; s++) {
                        const uint32_t bit = 1u << s;
                        if (L + 1 < p.n_layers) {
                            mbar_expect_tx(smem_u32(&sh->rx[s]), STG_BYTES);
                            ok = mbar_wait_cluster(smem_u32(&sh->rx[s]), (rx_par >> s) & 1, abort_flag, p.err, FFCU_ERR_EPI_TIMEOUT, p.wait_cycles);
                            rx_par ^= bit;
                        } else {                              // nothing comes; not before the layer's own phase has begun, though
                            ok = mbar_wait(smem_u32(&sh->face_done[s]), (uint32_t)i & 1, abort_flag, p.err, FFCU_ERR_EPI_TIMEOUT, p.wait_cycles);
                        }
                        if (ok) mbar_arrive_release_cluster(leader_ready + (uint32_t)(s * 8));
                    }
                }
            }
        }
    } else if (warp == TC_ISSUER2_WARP) {
        // Faces' first inputs (a slot is free once its last face's MMAs are done) and the fused BNs' byte tables.  Waits only where the
        // next phase needs what it does then: a parity says nothing about a phase that is two ahead, and the accumulators', which do
        // not wait for this warp in a PReLU layer, could be.
        const uint32_t a0_leader = map_to_cta(smem_u32(&sh->a0_full[0]), 0);
        auto load_face = [&](int s, int j) {                  // the pair's j-th face
            if (lane == 0) {
                if (rank == 0) mbar_expect_tx(smem_u32(&sh->a0_full[s]), 2 * ACT_BYTES);
#pragma unroll
                for (int pl = 0; pl < 2; pl++)
                    tma2_load_4d(s0 + s * ACT_BYTES + pl * PLANE_BYTES, &mapA, a0_leader + s * 8, pl * 128, -1, (int)rank * 7 - 1, p.face0 + pair + j * n_pairs);
            }
            __syncwarp();
        };
        const long long hold = rank == 0 ? p.hold_cycles : 0;
        uint32_t lut_par = 0;
        bool ok = true;
        tc_pdl_wait();
        tc_hold(hold);
        for (int j = 0; j < 2 && j < nf; j++) load_face(j, j);
#pragma unroll 1
        for (int i = 0; i < rounds && ok; i++) {
#pragma unroll 1
            for (int L = 0; L < p.n_layers && ok; L++) {
                const uint8_t* lut = p.layers[L].lut;
                if (!lut) continue;
                // (twice the limit: whoever this wait depends on gives up first, and says where)
                ok = mbar_wait(smem_u32(&sh->lut_empty), lut_par ^ 1, abort_flag, p.err, FFCU_ERR_EMPTY_TIMEOUT, 2 * p.wait_cycles);
                lut_par ^= 1;
                if (ok && lane == 0) {
                    mbar_expect_tx(smem_u32(&sh->lut_full), LUT_BYTES);
                    bulk_load(s0 + OFF_LUT, lut + rank * LUT_BYTES, LUT_BYTES, smem_u32(&sh->lut_full));
                }
                __syncwarp();
                tc_hold(hold);
            }
#pragma unroll 1
            for (int s = 0; s < 2 && ok; s++) {
                const int j = 2 * (i + 1) + s;
                if (j >= nf) break;
                ok = mbar_wait(smem_u32(&sh->face_done[s]), (uint32_t)i & 1, abort_flag, p.err, FFCU_ERR_EPI_TIMEOUT, 2 * p.wait_cycles);
                if (ok) load_face(s, j);
            }
        }
    } else {
        FaceEpi e;
        e.rank = (int)rank; e.peer = rank ^ 1u; e.lane = lane; e.q = warp & 3; e.g = warp >> 2;
        e.ch = e.q * 32 + lane;
        e.row_tx = (rank ? 0 : 6) + 2 * e.g;
        e.hr_own = (rank ? 16 : 0) + 3 * e.g;
        e.lut_lo = (uint32_t)(lane * 4 + (e.q & 1) * 128) * 0x01010101u;
        e.lut_hi = (uint32_t)(e.q >> 1) * 0x01010101u;
        const uint32_t leader_ready = map_to_cta(smem_u32(&sh->in_ready[0]), 0);
        uint32_t acc_par = 0, lut_par = 0;
        bool ok = true;
        tc_pdl_wait();
#pragma unroll 1
        for (int i = 0; i < rounds; i++) {
            const int slots = nf - 2 * i < 2 ? 1 : 2;
#pragma unroll 1
            for (int L = 0; L < p.n_layers; L++) {
                const FaceLayer* cl = p.layers + L;
                const float4 k = __ldg(cl->tab + rank * 128 + e.ch);
                const bool bn = cl->lut != nullptr;
                const bool last = L + 1 == p.n_layers;
                if (last && i + 1 == rounds && warp == 0) tc_pdl_trigger();
#pragma unroll 1
                for (int s = 0; s < slots; s++) {
                    const int face = p.face0 + pair + (2 * i + s) * n_pairs;
                    const uint32_t par = (acc_par >> s) & 1;
                    acc_par ^= 1u << s;
                    if (last)    face_epilogue<CONTRACT, true, true>(smem, sh, e, cl, k, s, face, tmem_base, par, leader_ready, s == 0, lut_par, abort_flag, p, ok);
                    else if (bn) face_epilogue<CONTRACT, true, false>(smem, sh, e, cl, k, s, face, tmem_base, par, leader_ready, s == 0, lut_par, abort_flag, p, ok);
                    else         face_epilogue<CONTRACT, false, false>(smem, sh, e, cl, k, s, face, tmem_base, par, leader_ready, false, lut_par, abort_flag, p, ok);
                }
                if (bn) {
                    lut_par ^= 1;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&sh->lut_empty));
                }
            }
        }
    }
    // teardown: neither CTA leaves while its partner may still write or read its memory
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
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

template <bool CONTRACT>
int set_smem()
{
    static int done[64] = {};             // per device: the attribute belongs to the device's copy of the function
    int dev = 0;
    FFCU_CHECK(cudaGetDevice(&dev));
    if (!done[dev & 63]) {
        FFCU_CHECK(cudaFuncSetAttribute(conv_face_kernel<CONTRACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_face_smem_bytes()));
        done[dev & 63] = 1;
    }
    return 0;
}

}  // namespace

int tc_face_smem_bytes() { return OFF_SH + (int)sizeof(FaceShared); }

int tc_launch_face(int mode, int pairs, cudaStream_t s, const CUtensorMap& mapA, const FaceParams& prm)
{
    const int rc = mode ? set_smem<true>() : set_smem<false>();
    if (rc != 0) return rc;
    return mode ? tc_launch_ex(conv_face_kernel<true>, 2 * pairs, tc_face_smem_bytes(), s, 2, mapA, prm)
                : tc_launch_ex(conv_face_kernel<false>, 2 * pairs, tc_face_smem_bytes(), s, 2, mapA, prm);
}

// How many pairs the device holds at once (0: none, or the attribute was refused).
int tc_face_pairs()
{
    if (set_smem<true>() != 0 || set_smem<false>() != 0) { cudaGetLastError(); return 0; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = tc_face_smem_bytes();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, conv_face_kernel<true>, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
    return n;
}
