// conv_tc_fc.cu -- the FC layer (512 outputs over K = 25088) as a split-K tensor-core GEMM.
//
// The weights are the MMA's rows: a tile is 128 outputs x up to 256 faces (N = the faces, rounded up to 16), so a small call
// moves and computes little for faces that are not there, and each weight passes through shared memory once per 256 faces.  A
// tile is cut into `splits` K ranges, one CTA each: 4 tiles x 28 ranges = 112 CTAs up to 256 faces, 7 K blocks of 128 each, all
// of them requested at once up to 128 faces (the weights before the programmatic-dependency wait).  A CTA lays its int32 partial sums
// [face][128 outputs] into shared memory as its threads hold them (a thread is an output: 32 lanes, 32 consecutive words),
// where a bulk reduction adds them to a scratch array (integer addition, so any order gives the same bits); the CTA that
// takes the last ticket of its tile turns the sums into floats exactly as the one-CTA form does (reference
// kernels/gemm_int8_matvec.c: out = (float)dot * w_scale + bias), leaving sums and ticket zero for the next call.
//
// Bound: latency (launch, fill, two L2 round trips for the hand-over), at 256 faces the 14.7 MB of additions.  Against tiles of
// 128 faces x 64 outputs with an atomic addition per sum, 5 / 17 / 33 / 64 / 128 / 256 / 512 faces: 9.0 / 14.1 / 20.0 / 20.0 / 20.2 /
// 24.3 / 33.2 -> 6.3 / 6.9 / 7.5 / 8.4 / 10.8 / 18.0 / 20.5 us.
#include "conv_tc_common.cuh"

#define FCT_KC 128
#define FCT_W_BYTES (128 * FCT_KC)

template <bool CONTRACT>
__global__ void __launch_bounds__(TC_THREADS, 1)
fc_tc_kernel(const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapW, const FcTcParams p)
{
    tc_pdl_trigger();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    TcShared* sh = (TcShared*)(smem + p.ring_bytes);
    __shared__ int s_last;
    const uint32_t tmem_cols = p.n_cols <= 32 ? 32 : p.n_cols <= 64 ? 64 : p.n_cols <= 128 ? 128 : 256;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    // CTA -> (tile of outputs, tile of faces, K range); the outputs vary fastest so that the CTAs of one K range (which read
    // the same activation boxes) are launched together
    const int tn = blockIdx.x % p.tiles_n;
    const int tm = (blockIdx.x / p.tiles_n) % p.tiles_m;
    const int split = blockIdx.x / (p.tiles_n * p.tiles_m);
    const int n_steps = p.blocks_per_split;
    const int kb0 = split * n_steps;
    const int sub = FCT_W_BYTES + p.n_cols * FCT_KC;             // a stage: weights, activations

    tc_setup(sh, p.stages, tmem_cols, warp, 4);
    const uint32_t tmem_base = sh->tmem_base;
    volatile int* abort_flag = &sh->abort_flag;
    const uint32_t full0 = smem_u32(&sh->full[0]), empty0 = smem_u32(&sh->empty[0]);

    if (warp == TC_PRODUCER_WARP) {
        // lanes 0 and 1: 64 rows of weights each, lane 2: the activations
        const uint32_t smem0 = smem_u32(smem) + (uint32_t)(lane * (FCT_W_BYTES / 2));
        const int pre = n_steps < p.stages ? n_steps : p.stages;
#pragma unroll 1
        for (int it = 0; it < pre; it++) {
            if (lane == 0) mbar_expect_tx(full0 + it * 8, (uint32_t)sub);
            __syncwarp();
            if (lane < 2) tma_load_4d(smem0 + it * sub, &mapW, full0 + it * 8, (kb0 + it) * FCT_KC, tn * 128 + lane * 64, 0, 0);
        }
        tc_pdl_wait();
        int stage = 0; uint32_t phase = 0;
        bool ok = true;
#pragma unroll 1
        for (int it = 0; it < n_steps && ok; it++) {
            if (it >= pre) {
                ok = mbar_wait(empty0 + stage * 8, phase ^ 1, abort_flag, p.err, FFCU_ERR_EMPTY_TIMEOUT, p.wait_cycles);
                if (!ok) break;
                if (lane == 0) mbar_expect_tx(full0 + stage * 8, (uint32_t)sub);
                __syncwarp();
                if (lane < 2) tma_load_4d(smem0 + stage * sub, &mapW, full0 + stage * 8, (kb0 + it) * FCT_KC, tn * 128 + lane * 64, 0, 0);
            }
            // (drop_step: armed by the timeout test for one launch, this step's activations never arrive)
            if (lane == 2 && it != p.drop_step)
                tma_load_4d(smem0 + stage * sub, &mapX, full0 + stage * 8, (kb0 + it) * FCT_KC, 0, 0, tm * p.n_cols);
            if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
    } else if (warp == TC_ISSUER_WARP) {
        if (tc_elect_one()) {
            const uint32_t idesc = idesc_i8(p.n_cols);
            int stage = 0; uint32_t phase = 0;
            bool ok = true;
            const uint64_t da0 = smem_desc<FCT_KC>(smem_u32(smem)), db0 = smem_desc<FCT_KC>(smem_u32(smem) + FCT_W_BYTES);
#pragma unroll 1
            for (int it = 0; it < n_steps; it++) {
                ok = mbar_wait(full0 + stage * 8, phase, abort_flag, p.err, FFCU_ERR_TMA_TIMEOUT, p.wait_cycles);
                if (!ok) break;
                tc_fence_after();
                const uint32_t soff = (uint32_t)((stage * sub) >> 4);
#pragma unroll
                for (int k = 0; k < FCT_KC / 32; k++)
                    umma_i8(tmem_base, da0 + (uint64_t)(soff + 2 * k), db0 + (uint64_t)(soff + 2 * k), idesc, (it | k) ? 1u : 0u);
                umma_commit(empty0 + stage * 8);
                if (++stage == p.stages) { stage = 0; phase ^= 1; }
            }
            if (ok) umma_commit(smem_u32(&sh->acc_full[0]));
        }
    } else if (warp < 16) {
        // Epilogue: a warp = (TMEM lane quarter: 32 outputs, every fourth 16 faces).  The ring's memory is idle once the
        // accumulator is complete: every MMA has read its operands and no copy is in flight.
        tc_pdl_wait();                                       // the scratch sums and tickets belong to the previous call until here
        const int q = warp & 3;
        const int f0 = tm * p.n_cols;                        // first face of the tile
        const int rows = p.batch - f0 < p.n_cols ? p.batch - f0 : p.n_cols;
        int* stg = (int*)smem;
        int* sums = p.sums + ((size_t)tn * p.batch + f0) * 128;
        const float4 ws = __ldg((const float4*)(p.w_scale + tn * 128) + lane), bi = __ldg((const float4*)(p.bias + tn * 128) + lane);
        const bool ok = mbar_wait(smem_u32(&sh->acc_full[0]), 0, abort_flag, p.err, FFCU_ERR_EPI_TIMEOUT, p.wait_cycles);
        if (ok) {
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
            for (int c = 16 * (warp >> 2); c < p.n_cols; c += 64) {
                int v[16];
                tmem_ld16_issue(taddr + (uint32_t)c, v);
                tmem_ld_wait(v);
#pragma unroll
                for (int i = 0; i < 16; i++) stg[(c + i) * 128 + q * 32 + lane] = v[i];
            }
            tc_fence_before();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        asm volatile("bar.sync 1, 512;" ::: "memory");
        // each warp sends a sixteenth of the faces; all are added (or the CTA has given up) before the ticket is taken
        const int per = (rows + 15) / 16, first = warp * per, count = rows - first < per ? rows - first : per;
        if (lane == 0 && count > 0 && !*abort_flag) {
            asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.s32 [%0], [%1], %2;"
                         ::"l"(sums + (size_t)first * 128), "r"(smem_u32(stg + first * 128)), "r"((uint32_t)(count * 512)) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
            asm volatile("fence.proxy.async;" ::: "memory");
            __threadfence();
        }
        asm volatile("bar.sync 1, 512;" ::: "memory");
        if (threadIdx.x == 0) {
            s_last = (!*abort_flag && atomicAdd(p.tickets + tm * p.tiles_n + tn, 1) == p.splits - 1) ? 1 : 0;
            __threadfence();                                 // the other CTAs' additions are visible from here on
        }
        asm volatile("bar.sync 1, 512;" ::: "memory");
        if (s_last) {
            __threadfence();
            // a warp takes a face, a lane four outputs of it; four faces' sums are requested before the first is used
#pragma unroll 1
            for (int r0 = warp; r0 < rows; r0 += 64) {
                int4 d[4];
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (r0 + 16 * k < rows) d[k] = __ldcg((const int4*)(sums + (size_t)(r0 + 16 * k) * 128) + lane);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int r = r0 + 16 * k;
                    if (r >= rows) break;
                    *((int4*)(sums + (size_t)r * 128) + lane) = make_int4(0, 0, 0, 0);       // clean for the next call
                    *((float4*)(p.out + (size_t)(f0 + r) * p.N + tn * 128) + lane) =
                        make_float4(ffcu_fc_fp<CONTRACT>(d[k].x, ws.x, bi.x), ffcu_fc_fp<CONTRACT>(d[k].y, ws.y, bi.y),
                                    ffcu_fc_fp<CONTRACT>(d[k].z, ws.z, bi.z), ffcu_fc_fp<CONTRACT>(d[k].w, ws.w, bi.w));
                }
            }
            if (threadIdx.x == 0) p.tickets[tm * p.tiles_n + tn] = 0;
        }
    }
    tc_teardown(abort_flag, tmem_base, tmem_cols, warp);
}

int tc_launch_fc(int mode, int grid, int smem, cudaStream_t s, const CUtensorMap& mapX, const CUtensorMap& mapW, const FcTcParams& prm)
{
    static int smem_set[64][2] = {};   // per device and instantiation: the attribute belongs to the device's copy of the function
    int dev = 0;
    FFCU_CHECK(cudaGetDevice(&dev));
    if (mode) {
        auto kern = fc_tc_kernel<true>;
        if (smem_set[dev & 63][1] < smem) {
            FFCU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            smem_set[dev & 63][1] = smem;
        }
        return tc_launch_ex(kern, grid, smem, s, 1, mapX, mapW, prm);
    }
    auto kern = fc_tc_kernel<false>;
    if (smem_set[dev & 63][0] < smem) {
        FFCU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        smem_set[dev & 63][0] = smem;
    }
    return tc_launch_ex(kern, grid, smem, s, 1, mapX, mapW, prm);
}
