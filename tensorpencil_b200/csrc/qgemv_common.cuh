// Pieces shared by the decode GEMV kernels (qgemv.cu, qgemv_mma.cu, qgemv_k.cu, qgemv_kmma.cu): the bounded
// mbarrier wait and the 1-D bulk copy that feed their shared-memory rings, packed f32 arithmetic and the field
// decoders of the GGUF formats.
#pragma once

#include <cuda_fp16.h>

#include "tpb_internal.h"

namespace tpb_gemv {

constexpr long long kWaitLimitCycles = 2000000000ll;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// Bounded wait: false when the limit ran out (status word written).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t *status,
                                          uint32_t code) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (uint32_t it = 0;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 255u) == 255u && clock64() - t0 > kWaitLimitCycles) {
            atomicCAS(status, 0u, code);
            return false;
        }
    }
}
// Exact int -> float for |v| < 2^22 on the ALU/FMA pipes: 0x4B400000 is 1.5 * 2^23 as a float, where
// one unit in the last place is 1, so adding v to the bit pattern adds v to the value.  The
// cvt instruction gives the same bits but issues at a quarter of the rate, which made it the
// limiter of the GEMVs with several activation rows (one conversion per block, row and column).
constexpr int kI2FMagicBits = 0x4B400000;
constexpr float kI2FMagic = 12582912.0f;
__device__ __forceinline__ float i2f_small(int v) { return __int_as_float(v + kI2FMagicBits) - kI2FMagic; }

// Untiled bulk copy global -> shared; both addresses and the size are multiples of 16 bytes.
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}


// Two packed f32 values; each half rounds like the scalar instruction.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float lo, float hi) {
    f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ f2 pack2i(int lo, int hi) {
    f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
    return d;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// Shared-memory loads by 32-bit shared address: one address register instead of a generic pointer pair.
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

// The weight rows [r0, r1) of warp gw of GW, for kernels that take them two at a time: contiguous and nearly equal, and dealt out in
// pairs where a warp gets more than one -- cut between any two rows, many warps end with a pair that is not full and costs a step all the same
// (14336 rows on 148 SMs x 14 warps: 6.92 rows a warp, four steps where 3.46 would do).
__device__ __forceinline__ void warp_row_pairs(int rows, int gw, int GW, int &r0, int &r1) {
    const int sh = rows > 2 * GW ? 1 : 0;
    const long long units = ((long long)rows + sh) >> sh;
    r0 = min(rows, (int)(units * gw / GW) << sh);
    r1 = min(rows, (int)(units * (gw + 1) / GW) << sh);
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// The two halves of a cluster barrier: every thread of every CTA of the cluster takes them in turn, a whole warp together.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

__device__ __forceinline__ float f16lo(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w & 0xffffu))); }
__device__ __forceinline__ float f16hi(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w >> 16))); }


enum { FMT_Q4_0 = 1, FMT_Q4_K = 2, FMT_Q5_K = 3, FMT_Q6_K = 4, FMT_IQ4_NL = 5 };

// Four 4-bit indices (one per byte of idx, 0..15) -> the four signed bytes of ggml's
// kvalues_iq4nl table: two byte-permutes over the table halves, merged by the index's bit 3.
__device__ __forceinline__ uint32_t iq4nl_lookup(uint32_t idx) {
    constexpr uint32_t T0 = 0xBFAD9881u;  // -127 -104 -83 -65
    constexpr uint32_t T1 = 0xF6EADDCFu;  // -49 -35 -22 -10
    constexpr uint32_t T2 = 0x26190D01u;  // 1 13 25 38
    constexpr uint32_t T3 = 0x71594535u;  // 53 69 89 113
    const uint32_t t = idx & 0x07070707u;
    const uint32_t u = t | (t >> 4);                     // byte 0: b0 | b1 << 4, byte 2: b2 | b3 << 4
    const uint32_t sel = __byte_perm(u, 0, 0x4420);      // 16-bit selector b0, b1, b2, b3
    const uint32_t v_lo = __byte_perm(T0, T1, sel);
    const uint32_t v_hi = __byte_perm(T2, T3, sel);
    const uint32_t m = ((idx >> 3) & 0x01010101u) * 0xffu;
    return (v_lo & ~m) | (v_hi & m);
}

// The 6-bit scales and mins of sub-blocks 2j and 2j+1 (j = 0..3) of a q4_k / q5_k super-block, both pairs at
// once and without a branch; s0, s1, s2 are the three words of the 12-byte scales field.  ggml's
// get_scale_min_k4 read two sub-blocks at a time: bytes 2j, 2j+1 of the field are one 16-bit word, and
//   j < 2:  scale = byte & 63 of word j of s0,              min = byte & 63 of word j of s1
//   j >= 2: scale = (s2 word & 0x0f0f) | (s0 word >> 6 << 4), min = (s2 word >> 4 & 0x0f0f) | (s1 word >> 6 << 4)
// with "word" the 16-bit half number (j & 1) of each 32-bit word.
__device__ __forceinline__ void scale_min_k4_pair(int j, uint32_t s0, uint32_t s1, uint32_t s2, float &sc0, float &mn0,
                                                  float &sc1, float &mn1) {
    const uint32_t sh = (uint32_t)(j & 1) * 16u;
    const uint32_t a = (s0 >> sh) & 0xffffu, b = (s1 >> sh) & 0xffffu, c = (s2 >> sh) & 0xffffu;
    const bool upper = j >= 2;
    const uint32_t s16 = upper ? ((c & 0x0f0fu) | ((a & 0xc0c0u) >> 2)) : (a & 0x3f3fu);
    const uint32_t m16 = upper ? (((c >> 4) & 0x0f0fu) | ((b & 0xc0c0u) >> 2)) : (b & 0x3f3fu);
    sc0 = (float)(s16 & 0xffu);
    sc1 = (float)(s16 >> 8);
    mn0 = (float)(m16 & 0xffu);
    mn1 = (float)(m16 >> 8);
}


}  // namespace tpb_gemv
