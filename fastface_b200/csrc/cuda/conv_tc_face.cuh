// conv_tc_face.cuh -- what the kernels that take a face through a stage share: the epilogue of one output channel per
// thread (weights are the MMA's rows, a row of the face 8, 16 or 32 of its columns).
#pragma once
#include "conv_tc_common.cuh"

#define FACE_LUT_BYTES (128 * 256)       // fused BN byte table of a CTA's 128 channels

__device__ __forceinline__ void mbar_arrive_release_cluster(uint32_t cluster_addr)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_ld8_issue(uint32_t taddr, int (&v)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait8(int (&v)[8])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]) :: "memory");
}
// MMAs issued so far are done: one arrival on this barrier of each CTA in `mask`.
__device__ __forceinline__ void umma_commit_multicast(uint32_t bar, uint16_t mask)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(mask) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Shared memory of this CTA -> a CTA of the cluster, counted on that CTA's barrier (all shared::cluster addresses but `from`).
__device__ __forceinline__ void bulk_send(uint32_t to, uint32_t from, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(to), "r"(from), "r"(bytes), "r"(bar) : "memory");
}

// What a thread's stores need: ad[k] = its byte's shared-memory address in a line of swizzle phase k of the row that is
// written (lines of 128 B: column c lies c + 1 lines further on, in phase (c + 1) & 7), or, in the last layer, the NHWC pixel.
struct FaceDst {
    uint32_t ad[8];
    int8_t* g;
};

// NV (four, or two at a row's end) positions c0 .. of one channel: accumulators v, constants k (w_scale, bias, PReLU slope or
// residual scale, inv_out) -> int8.  rw: the residual's bytes in, the requantised ones out.  What the next layer reads (the
// fused BN of it, where the layer has one) is stored byte by byte: a warp's 32 channels are 32 consecutive bytes of a line.
// lut_lo, lut_hi: this channel's share of a table address, in every byte; entry q of channel 32 * quarter + lane lies at
// (q >> 2) * 512 + quarter * 128 + lane * 4 + (q & 3) of the table, so 32 lanes never meet in a bank.
template <bool CONTRACT, bool RESBN, int NV>
__device__ __forceinline__ uint32_t face_quad(const int* v, uint32_t rw, const float4& k)
{
    int q[4] = {0, 0, 0, 0};
    const uint32_t rx = rw ^ 0x80808080u;
    TcUnroll<NV>::run([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        const float f = ffcu_conv_fp_f<CONTRACT>(__int2float_rn(v[i]), k.x, k.y, RESBN, RESBN ? ffcu_byte2f<i>(rx) : 0.0f, k.z, !RESBN, k.z);
        q[i] = ffcu_requant_nosat<false>(f, k.w);
    });
    return (uint32_t)ffcu_pack4(q[0], q[1], q[2], q[3]);
}
template <bool CONTRACT, bool RESBN, bool LAST, int C0, int C1, int ROW, int W = 14, int C = FACE_C, int PITCH = 16>
__device__ __forceinline__ void face_cols(const int* v, uint32_t* rw, const float4& k, const uint8_t* lut, uint32_t lut_lo,
                                          uint32_t lut_hi, const FaceDst& d)
{
    constexpr int N = C1 - C0, WORDS = (N + 3) / 4;
    TcUnroll<WORDS>::run([&](auto gc) {
        constexpr int g = decltype(gc)::value;
        rw[g] = face_quad<CONTRACT, RESBN, (N - 4 * g < 4 ? N - 4 * g : 4)>(v + 4 * g, rw[g], k);
    });
    uint32_t b[N];
    TcUnroll<N>::run([&](auto ic) {
        constexpr int i = decltype(ic)::value, m = i & 3;
        const uint32_t w = rw[i / 4];
        if constexpr (RESBN) {
            const uint32_t lo = (w & 0x03030303u) | lut_lo, hi = ((w >> 1) & 0x7e7e7e7eu) | lut_hi;
            uint32_t off;            // byte 0: lo, byte 1: hi, above it hi's sign (zero)
            asm("prmt.b32 %0, %1, %2, %3;" : "=r"(off) : "r"(hi), "r"(lo), "n"(((m | 8) << 12) | ((m | 8) << 8) | (m << 4) | (4 + m)));
            b[i] = lut[off];
        } else b[i] = w >> (8 * m);
    });
    TcUnroll<N>::run([&](auto ic) {
        constexpr int i = decltype(ic)::value, c = C0 + i;
        if constexpr (LAST) d.g[(ROW * W + c) * C] = (int8_t)b[i];
        else asm volatile("st.shared.u8 [%0 + %1], %2;" ::"r"(d.ad[(c + 1) & 7]), "n"(ROW * PITCH * 128 + (c + 1) * 128), "r"(b[i]));
    });
}
template <bool CONTRACT, bool RESBN, bool LAST, int ROW>
__device__ __forceinline__ void face_half_a(const int* v, uint32_t* rw, const float4& k, const uint8_t* lut, uint32_t lo, uint32_t hi, const FaceDst& d)
{
    face_cols<CONTRACT, RESBN, LAST, 0, 8, ROW>(v, rw, k, lut, lo, hi, d);
}
template <bool CONTRACT, bool RESBN, bool LAST, int ROW>
__device__ __forceinline__ void face_half_b(const int* v, uint32_t* rw, const float4& k, const uint8_t* lut, uint32_t lo, uint32_t hi, const FaceDst& d)
{
    face_cols<CONTRACT, RESBN, LAST, 8, 14, ROW>(v, rw, k, lut, lo, hi, d);
}

