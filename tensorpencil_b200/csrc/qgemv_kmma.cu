// Decode GEMV for the GGUF formats q4_0, iq4_nl, q4_k, q5_k and q6_k on mma.sync, for several activation rows (sm_100a).
//
// Why: the dp4a kernels (qgemv_k.cu) decode a lane's weights and then spend one dp4a per weight word and activation
// row; from a few activation rows on they are bound by instruction issue, not by HBM.  Here sixteen weight rows are the m
// side of mma.sync.m16n8k32 (k16 for q6_k, whose scales cover 16 elements) and the activation rows its n side: one
// decode of the quants into A fragments and one instruction per 512 weights serve all eight activation rows.
//
// Same bits as the dp4a kernels, so that a row's result depends neither on its group nor on the kernel that took it.  There, lane l
// adds the terms of units (64 elements) l, l + 32, l + 64, .. in order and a butterfly adds the lanes.  Here consumer warp w of
// sixteen takes units w, w + 16, w + 32, ..: the even ones of them are lane w's, the odd ones lane (w + 16)'s, kept in two accumulators with
// the same operations in the same order; their sum is the butterfly's first step, and the sixteen warps' sums are added in the
// order of its other four.  That a warp's units are 16 apart also makes everything but the base address of a stage a constant
// of the warp: quarter or half of a super-block, shifts, offsets.
//
// Layout.  One CTA per SM owns a contiguous range of weight rows and streams them in stages of 16 rows with 1-D bulk copies through a
// ring that fills shared memory; four producer warps issue them, before griddepcontrol.wait (weights are constants).  K goes by
// in passes of at most 6 units per warp, whose activations a warp keeps as B fragments in registers; with more than one
// pass the accumulators of a few row groups wait in shared memory between passes.  Activation block scales and the terms of the
// formats' offsets (dx * sum(xq)) are in a table of the warp's own, and so are the decoded scales of a stage, one task per
// row and unit: decoded unit pair by unit pair, with a warp barrier around each, they broke the warp's work into short
// dependent chains (q4_k 17408 x 5120, 20 -> 17.5 us without).
//
// What bounds it: latency within a warp -- twenty warps, four to a scheduler with 96 registers each, issue in half of the cycles, and
// the reads of scales and tables keep the shared-memory pipe 45 % busy (ncu, q4_k 17408 x 5120); the tensor pipe is at 5 %.  So a
// launch costs nearly the same whatever the number of activation rows is: q4_k 17408 x 5120 17.0 us at M = 1, 18.1 at 8 (floor 7.8),
// where the dp4a kernel takes 12.5 and 32.2.  us at M = 8, dp4a / here: 5120 x 17408 q4_k 56 / 27, q5_k 65 / 31, q6_k 87 / 43;
// 17408 x 5120 q5_k 35 / 23, q6_k 45 / 29; 32000 x 4096 q4_k 52 / 23; 4096 x 14336 q4_0 39 / 18, iq4_nl 50 / 24.  The dispatch rule
// is mma_wins in qgemv_k.cu.
//
// Rows of a stage are `pitch` bytes apart with pitch = 48 mod 128: the eight rows of a fragment load (8 x 16 or
// 4 x 32 bytes at a time) then fall on distinct banks.
//
// Block layouts: src/core/quants.zig:9-16 (ggml's).  Reference kernels these stand in for: src/gpu/cuda/elt.zig:2014-2110,
// :1831-1925, :1526-1713, :1714-1830, dispatched from Backend.opGemvQuantQ8N (src/gpu/cuda/backend.zig:1719-1735).
#include <cuda_fp16.h>

#include <type_traits>

#include "qgemv_common.cuh"

using namespace tpb_gemv;

namespace {

constexpr int kConsumers = 16;     // fixed by the order of the sums
constexpr int kProducers = 4;      // twenty warps in all: from seventeen on a thread has 96 registers
constexpr int kThreads = 32 * (kConsumers + kProducers);
constexpr int kRows = 16;          // weight rows of a stage = m of the MMA
constexpr int kPart = kRows * 8;   // floats of one warp's sums
constexpr int NU = 6;              // units of a pass per consumer warp (four registers of activations each)
constexpr int kSwBytes = NU * 256; // decoded scales of a warp: 16 bytes per unit and row

// bytes of a super-block of 256 elements
__host__ __device__ constexpr int sb_bytes(int fmt) {
    return fmt == FMT_Q5_K ? 176 : fmt == FMT_Q6_K ? 210 : 144;
}
// activation table, per unit: [2 blocks][4 t]{dx, dx, S, S}; q6_k [4 runs][4 t]{dx, dx, T, T}
__host__ __device__ constexpr int tab_bytes(int fmt) { return fmt == FMT_Q6_K ? 256 : 128; }

struct KmmaParams {
    float *y;
    const uint8_t *w;
    const float *xd;   // activation block scales [m][nblk]
    const int8_t *xq;  // activation quants [m][cols]
    float scale;
    int rows, cols, nblk, m;
    int npass;         // passes over K, of whole groups of 4 super-blocks (16 units: one per consumer warp)
    int blk_rg;        // row groups whose accumulators are kept between passes (npass > 1)
    int pitch;         // bytes between the rows of a stage
    int stages;
    uint32_t row_bytes;
    uint32_t *status;
};

// C (16 weight rows x 8 activation rows) = c_in + A (16 x 32 unsigned bytes) * B (32 x 8 signed bytes).
// Lane (g = lane / 4, t = lane % 4): a0 / a2 = row g, a1 / a3 = row g + 8; c0, c1 = row g, columns 2t, 2t + 1; c2, c3 = row g + 8.
template <bool SIGNED_A>
__device__ __forceinline__ void mma_k32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1,
                                        int ci0, int ci1) {
    if (SIGNED_A)
        asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%10,%11};"
            : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(ci0), "r"(ci1));
    else
        asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%10,%11};"
            : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(ci0), "r"(ci1));
}
__device__ __forceinline__ void mma_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0, int ci0, int ci1) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%7,%8};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(b0), "r"(ci0), "r"(ci1));
}

__device__ __forceinline__ uint2 lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void lds_2f2(uint32_t addr, f2 &a, f2 &b) {
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}
__device__ __forceinline__ float4 lds_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, float a, float b, float c, float d) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
    return v;
}

template <int FMT>
__global__ void __launch_bounds__(kThreads, 1) kquant_gemv_mma_kernel(const KmmaParams p) {
    constexpr bool Q4 = FMT == FMT_Q4_0 || FMT == FMT_IQ4_NL;
    constexpr bool Q6 = FMT == FMT_Q6_K;
    constexpr int kSb = sb_bytes(FMT);
    extern __shared__ __align__(128) uint8_t smem[];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int S = p.stages;
    const int stage_bytes = kRows * p.pitch;
    const int n_sb = p.cols / 256;
    const int n_grp4 = (n_sb + 3) / 4;      // groups of 4 super-blocks; the last may be partial

    // shared: [ring][activation tables][decoded scales][parts: 2 x 16 warps][barriers][accumulators between passes]
    const uint32_t ring = smem_u32(smem);
    const uint32_t tab = ring + (uint32_t)(S * stage_bytes) + (uint32_t)(warp * NU * tab_bytes(FMT));
    const uint32_t sw = ring + (uint32_t)(S * stage_bytes + kConsumers * NU * tab_bytes(FMT) + warp * kSwBytes);
    float *s_part = reinterpret_cast<float *>(smem + (size_t)S * stage_bytes + (size_t)kConsumers * (NU * tab_bytes(FMT) + kSwBytes));
    const uint32_t bars = smem_u32(s_part + 2 * kConsumers * kPart);
    float *s_acc = s_part + 2 * kConsumers * kPart + 40;     // [blk_rg][16 warps][2 accumulators][kPart]
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (S + s); };
    auto pfull_bar = [&](int b) { return bars + 8u * (2 * S + b); };
    auto pempty_bar = [&](int b) { return bars + 8u * (2 * S + 2 + b); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(full_bar(s)), "r"(kProducers));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty_bar(s)), "r"(kConsumers));
        }
        for (int b = 0; b < 2; b++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(pfull_bar(b)), "r"(kConsumers));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(pempty_bar(b)), "r"(1));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const int r_begin = (int)((long long)p.rows * blockIdx.x / gridDim.x);
    const int r_end = (int)((long long)p.rows * (blockIdx.x + 1) / gridDim.x);
    const int n_rg = (r_end - r_begin + kRows - 1) / kRows;
    const int blk_rg = p.npass > 1 ? p.blk_rg : n_rg;
    const int total = n_rg * p.npass;       // stages, in the order block of row groups, pass, row group
    // super-blocks of a pass: whole groups of 4, but for the row's end
    auto pass_sb = [&](int pass) { return min(n_sb, n_grp4 * pass / p.npass * 4); };

    if (warp >= kConsumers) {
        // ---------------- producers ----------------
        const int pw = warp - kConsumers;
        const int r = pw * (kRows / kProducers) + lane;     // this lane's row of a stage
        int is_b0 = 0, is_rg = 0, is_pass = 0, is_slot = 0;
        auto issue = [&]() {
            const int sb0 = pass_sb(is_pass), sb1 = pass_sb(is_pass + 1);
            const int row = r_begin + is_rg * kRows + r;
            const bool mine = lane < kRows / kProducers && row < r_end;
            size_t off = (size_t)row * p.row_bytes + (size_t)sb0 * kSb;
            uint32_t bytes = (uint32_t)(sb1 - sb0) * kSb;
            if (Q6) {
                // super-blocks of 210 bytes: copy from the 16-byte boundary below, up to the one that ends the
                // 16-byte word of the last byte; the row then sits `mis` bytes into its slot
                const uint32_t mis = (uint32_t)off & 15u;
                off -= mis;
                bytes = (bytes + mis + 15u) & ~15u;
            }
            const uint32_t tx = __reduce_add_sync(0xffffffffu, mine ? bytes : 0u);
            const uint32_t bar = full_bar(is_slot);
            if (lane == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(tx) : "memory");
            __syncwarp();
            if (mine) bulk_g2s(ring + (uint32_t)(is_slot * stage_bytes + r * p.pitch), p.w + off, bytes, bar);
            if (++is_slot == S) is_slot = 0;
            if (++is_rg == min(is_b0 + blk_rg, n_rg)) {
                is_rg = is_b0;
                if (++is_pass == p.npass) {
                    is_pass = 0;
                    is_b0 += blk_rg;
                    is_rg = is_b0;
                }
            }
        };
        for (int i = 0; i < S && i < total; i++) issue();
        asm volatile("griddepcontrol.wait;" ::: "memory");
        int slot = 0, b0 = 0, pass = 0, rg = 0, done = 0;
        uint32_t par = 0;
        for (int j = 0; j < total; j++) {
            bool ok = true;
            if (pw == 0 || j + S < total) ok = mbar_wait(empty_bar(slot), par, p.status, (11u << 24) | (uint32_t)slot);
            if (!__all_sync(0xffffffffu, ok)) break;
            if (j + S < total) {
                // order the consumers' generic-proxy reads of the slot before the async-proxy refill
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                issue();
            }
            if (pw == 0 && pass == p.npass - 1) {
                // a row group is done: add the warps' sums, as the butterfly's steps 8, 4, 2, 1 would
                const int b = done & 1;
                ok = mbar_wait(pfull_bar(b), (uint32_t)(done >> 1) & 1u, p.status, (11u << 24) | 0x100u | (uint32_t)b);
                if (!__all_sync(0xffffffffu, ok)) break;
                const float *part = s_part + (size_t)b * kConsumers * kPart + 4 * lane;
                float4 v[8];
#pragma unroll
                for (int w = 0; w < 8; w++) {
                    const float4 lo = *reinterpret_cast<const float4 *>(part + w * kPart), hi = *reinterpret_cast<const float4 *>(part + (w + 8) * kPart);
                    v[w] = make_float4(lo.x + hi.x, lo.y + hi.y, lo.z + hi.z, lo.w + hi.w);
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1)
#pragma unroll
                    for (int w = 0; w < o; w++)
                        v[w] = make_float4(v[w].x + v[w + o].x, v[w].y + v[w + o].y, v[w].z + v[w + o].z, v[w].w + v[w + o].w);
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(pempty_bar(b)) : "memory");
                const int row = r_begin + rg * kRows + (lane >> 2), c = 2 * (lane & 3);
                const float v4[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int rr = row + (e >> 1) * 8, cc = c + (e & 1);
                    if (rr < r_end && cc < p.m) p.y[(size_t)cc * p.rows + rr] = v4[e] * p.scale;
                }
                done++;
            }
            if (++slot == S) {
                slot = 0;
                par ^= 1u;
            }
            if (++rg == min(b0 + blk_rg, n_rg)) {
                rg = b0;
                if (++pass == p.npass) {
                    pass = 0;
                    b0 += blk_rg;
                    rg = b0;
                }
            }
        }
        return;
    }

    // ---------------- consumers: units warp, warp + 16, .. of a row ----------------
    const int g = lane >> 2, t = lane & 3;
    const f2 magic2 = pack2(kI2FMagic, kI2FMagic);
    // what all of a warp's units share: quarter (q6_k: half and run) of the super-block, and its offset in a group of 4
    const int jj = warp & 3;
    const uint32_t sb_off = (uint32_t)((warp >> 2) * kSb);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int slot = 0, done = 0;
    uint32_t par = 0;
    for (int b0 = 0; b0 < n_rg; b0 += blk_rg)
    for (int pass = 0; pass < p.npass; pass++) {
        const int sb0 = pass_sb(pass), pass_units = 4 * (pass_sb(pass + 1) - sb0);
        const int nu = (pass_units - warp + 15) >> 4;                  // this warp's units of the pass, <= NU (checked by the host)
        const int gu0 = 4 * sb0 + warp;                                // the first of them within the row
        // The first unit of the pass belongs to lane (warp)'s sum where sb0 / 4 is even: accumulator (sb0 / 4 + u) & 1.  The two
        // are swapped on the way in and out instead.
        const int swap = (sb0 >> 2) & 1;
        // B fragments: a lane loads 16 contiguous activations of its unit (for q6_k the run p = t of 16), makes their table entry,
        // and the quad exchanges words.
        // (All loads first: behind the table's stores each block scale would cost a round trip to L2 of its own.)
        uint32_t b[NU][4];
        {
            float dl[NU];
            __syncwarp();
#pragma unroll
            for (int u = 0; u < NU; u++) {
                b[u][0] = b[u][1] = b[u][2] = b[u][3] = 0u;
                dl[u] = 0.0f;
                if (u < nu && g < p.m) {
                    const int gu = gu0 + 16 * u;
                    dl[u] = __ldcg(p.xd + (size_t)g * p.nblk + (Q6 ? 4 * (gu >> 1) + t : 2 * gu + (t >> 1)));
                    const int e = Q6 ? 128 * (gu >> 1) + 32 * t + 16 * (gu & 1) : 64 * gu + 16 * t;
                    const uint4 v = __ldcg(reinterpret_cast<const uint4 *>(p.xq + (size_t)g * p.cols + e));
                    b[u][0] = v.x; b[u][1] = v.y; b[u][2] = v.z; b[u][3] = v.w;
                }
            }
#pragma unroll
            for (int u = 0; u < NU; u++) {
                if (u < nu) {
                    const float dx = dl[u];
                    int s = __dp4a((int)b[u][0], 0x01010101, 0);
                    s = __dp4a((int)b[u][1], 0x01010101, s);
                    s = __dp4a((int)b[u][2], 0x01010101, s);
                    s = __dp4a((int)b[u][3], 0x01010101, s);
                    if (!Q6) s += __shfl_xor_sync(0xffffffffu, s, 1);
                    if (Q6 || (t & 1) == 0) {
                        const uint32_t a = tab + (uint32_t)(u * tab_bytes(FMT) + (Q6 ? t : t >> 1) * 64 + (g >> 1) * 16 + (g & 1) * 4);
                        const float off = Q6 ? 32.0f * (dx * (float)s) : dx * (float)s;
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(dx) : "memory");
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(a + 8u), "f"(off) : "memory");
                    }
                    const bool hi2 = (t & 2) != 0, hi1 = (t & 1) != 0;
                    const uint32_t x0 = hi2 ? b[u][0] : b[u][2], x1 = hi2 ? b[u][1] : b[u][3];
                    const uint32_t y0 = __shfl_xor_sync(0xffffffffu, x0, 2), y1 = __shfl_xor_sync(0xffffffffu, x1, 2);
                    if (hi2) { b[u][0] = y0; b[u][1] = y1; } else { b[u][2] = y0; b[u][3] = y1; }
                    // q4_k, q5_k: lanes 0, 1 held the halves of the first block, lanes 2, 3 those of the second; lane t now has elements
                    // 8 (t >> 1) + 16 (t & 1) .. + 7 of both.  The other formats: word j of lane t -> word t of lane j.
                    if (Q4 || Q6) {
                        const uint32_t z0 = __shfl_xor_sync(0xffffffffu, hi1 ? b[u][0] : b[u][1], 1);
                        const uint32_t z1 = __shfl_xor_sync(0xffffffffu, hi1 ? b[u][2] : b[u][3], 1);
                        if (hi1) { b[u][0] = z0; b[u][2] = z1; } else { b[u][1] = z0; b[u][3] = z1; }
                    }
                }
            }
            __syncwarp();
        }

        for (int rg = b0; rg < min(b0 + blk_rg, n_rg); rg++) {
            bool ok = mbar_wait(full_bar(slot), par, p.status, (12u << 24) | (uint32_t)slot);
            if (!__all_sync(0xffffffffu, ok)) return;
            const uint32_t stage = ring + (uint32_t)(slot * stage_bytes);
            // a lane's rows g and g + 8, and as decoder row lane & 15: this warp's first unit
            uint32_t base_g = stage + (uint32_t)(g * p.pitch) + sb_off, base_h = base_g + (uint32_t)(8 * p.pitch);
            uint32_t base_r = stage + (uint32_t)((lane & 15) * p.pitch) + sb_off + (uint32_t)((lane >> 4) * 4 * kSb);
            if (Q6) {
                const uint32_t m0 = (uint32_t)(r_begin + rg * kRows) * p.row_bytes + (uint32_t)(sb0 * kSb);
                base_g += (m0 + (uint32_t)g * p.row_bytes) & 15u;
                base_h += (m0 + (uint32_t)(g + 8) * p.row_bytes) & 15u;
                base_r += (m0 + (uint32_t)(lane & 15) * p.row_bytes) & 15u;
            }
            f2 acc[2][2];       // [accumulator][rows g, g + 8]
            f2 *keep = reinterpret_cast<f2 *>(s_acc + ((size_t)((rg - b0) * kConsumers + warp) * 2) * kPart + 4 * lane);
            acc[0][0] = acc[0][1] = acc[1][0] = acc[1][1] = 0ull;
            if (pass > 0) {
                const ulonglong2 a0 = *reinterpret_cast<const ulonglong2 *>(keep + (swap ? kPart / 2 : 0));
                const ulonglong2 a1 = *reinterpret_cast<const ulonglong2 *>(keep + (swap ? 0 : kPart / 2));
                acc[0][0] = a0.x; acc[0][1] = a0.y;
                acc[1][0] = a1.x; acc[1][1] = a1.y;
            }
            // N: how many units, where it is known (the branches between units then go, and loads move ahead of the arithmetic)
            auto multiply = [&](auto n_tag) {
                constexpr int N = decltype(n_tag)::value;
                const int n_here = N ? N : nu;
            if constexpr (!Q4) {
                // the scales of all this warp's units first: lane = (unit & 1) * 16 + row
#pragma unroll
                for (int grp = 0; grp < NU / 2; grp++) {
                    if (2 * grp + (lane >> 4) < n_here) {
                        const uint32_t dst = sw + (uint32_t)(grp * 512 + lane * 16);
                        const uint32_t o = base_r + (uint32_t)(grp * 8 * kSb);
                        if constexpr (Q6) {
                            const float d = __half2float(__ushort_as_half((unsigned short)lds_u16(o + 208)));
                            const uint32_t so = o + 192u + 8u * (uint32_t)((warp >> 1) & 1);
                            float ws[4];
#pragma unroll
                            for (int q = 0; q < 4; q++) ws[q] = d * (float)(int)(int8_t)(lds_u16(so + 2 * q) >> (8 * (warp & 1)));
                            sts128(dst, ws[0], ws[1], ws[2], ws[3]);
                        } else {
                            const uint4 hdr = lds128(o);
                            const float d = f16lo(hdr.x), dmin = f16hi(hdr.x);
                            float sc0, mn0, sc1, mn1;
                            scale_min_k4_pair(jj, hdr.y, hdr.z, hdr.w, sc0, mn0, sc1, mn1);
                            sts128(dst, d * sc0, -(dmin * mn0), d * sc1 * (FMT == FMT_Q5_K ? 1.0f : 0.0625f), -(dmin * mn1));
                        }
                    }
                }
                __syncwarp();
            }
#pragma unroll
            for (int grp = 0; grp < NU / 2; grp++) {
                if (N == 0 && 2 * grp >= nu) break;
#pragma unroll
                for (int uu = 0; uu < 2; uu++) {
                    const int u = 2 * grp + uu;
                    if (u < n_here) {
                        f2 &ag_ = acc[uu][0], &ah_ = acc[uu][1];
                        const uint32_t swg = sw + (uint32_t)(u * 256 + g * 16);
                        const uint32_t ta = tab + (uint32_t)(u * tab_bytes(FMT) + t * 16);
                        if constexpr (Q4) {
                            // unit = two 18-byte blocks: f16 d, 16 nibble bytes (byte j: elements j and j + 16)
                            const uint32_t ag = base_g + (uint32_t)(u * 4 * kSb + jj * 36), ah = base_h + (uint32_t)(u * 4 * kSb + jj * 36);
                            const uint32_t g0 = lds32(ag), g4 = lds32(ag + 16), h0 = lds32(ah), h4 = lds32(ah + 16);
                            const uint32_t gw0 = lds32(ag + 4 * t), gw1 = lds32(ag + 4 * t + 4), gw2 = lds32(ag + 4 * t + 20);
                            const uint32_t hw0 = lds32(ah + 4 * t), hw1 = lds32(ah + 4 * t + 4), hw2 = lds32(ah + 4 * t + 20);
                            f2 dx0, s0, dx1, s1;
                            lds_2f2(ta, dx0, s0);
                            lds_2f2(ta + 64, dx1, s1);
                            const uint32_t ga = __funnelshift_r(gw0, gw1, 16), ha = __funnelshift_r(hw0, hw1, 16);
                            int c[4], e[4];
                            if (FMT == FMT_Q4_0) {
                                mma_k32<false>(c, ga & 0x0f0f0f0fu, ha & 0x0f0f0f0fu, (ga >> 4) & 0x0f0f0f0fu, (ha >> 4) & 0x0f0f0f0fu, b[u][0],
                                               b[u][1], kI2FMagicBits, kI2FMagicBits);
                                mma_k32<false>(e, gw2 & 0x0f0f0f0fu, hw2 & 0x0f0f0f0fu, (gw2 >> 4) & 0x0f0f0f0fu, (hw2 >> 4) & 0x0f0f0f0fu,
                                               b[u][2], b[u][3], kI2FMagicBits, kI2FMagicBits);
                            } else {
                                mma_k32<true>(c, iq4nl_lookup(ga & 0x0f0f0f0fu), iq4nl_lookup(ha & 0x0f0f0f0fu), iq4nl_lookup((ga >> 4) & 0x0f0f0f0fu),
                                              iq4nl_lookup((ha >> 4) & 0x0f0f0f0fu), b[u][0], b[u][1], kI2FMagicBits, kI2FMagicBits);
                                mma_k32<true>(e, iq4nl_lookup(gw2 & 0x0f0f0f0fu), iq4nl_lookup(hw2 & 0x0f0f0f0fu), iq4nl_lookup((gw2 >> 4) & 0x0f0f0f0fu),
                                              iq4nl_lookup((hw2 >> 4) & 0x0f0f0f0fu), b[u][2], b[u][3], kI2FMagicBits, kI2FMagicBits);
                            }
                            const float dg0 = f16lo(g0), dg1 = f16hi(g4), dh0 = f16lo(h0), dh1 = f16hi(h4);
                            ag_ = fma2(pack2(dg0, dg0), mul2(dx0, sub2(pack2i(c[0], c[1]), magic2)), ag_);
                            ah_ = fma2(pack2(dh0, dh0), mul2(dx0, sub2(pack2i(c[2], c[3]), magic2)), ah_);
                            if (FMT == FMT_Q4_0) {
                                ag_ = fma2(pack2(-8.0f * dg0, -8.0f * dg0), s0, ag_);
                                ah_ = fma2(pack2(-8.0f * dh0, -8.0f * dh0), s0, ah_);
                            }
                            ag_ = fma2(pack2(dg1, dg1), mul2(dx1, sub2(pack2i(e[0], e[1]), magic2)), ag_);
                            ah_ = fma2(pack2(dh1, dh1), mul2(dx1, sub2(pack2i(e[2], e[3]), magic2)), ah_);
                            if (FMT == FMT_Q4_0) {
                                ag_ = fma2(pack2(-8.0f * dg1, -8.0f * dg1), s1, ag_);
                                ah_ = fma2(pack2(-8.0f * dh1, -8.0f * dh1), s1, ah_);
                            }
                        } else if constexpr (Q6) {
                            // half n and run lh of the super-block; 4 bytes of each of the three fields per lane
                            const uint32_t n = (uint32_t)(warp >> 1) & 1u, fld = (uint32_t)(u * 4 * kSb) + 16u * (uint32_t)(warp & 1) + 4u * t;
                            const uint32_t og = base_g + fld, oh = base_h + fld;
                            const uint32_t sg = (og & 2u) * 8u, sh = (oh & 2u) * 8u;
                            const uint32_t lg = (og & ~3u) + 64u * n, lh = (oh & ~3u) + 64u * n;
                            const uint32_t qg = (og & ~3u) + 128u + 32u * n, qh = (oh & ~3u) + 128u + 32u * n;
                            const uint32_t gla = __funnelshift_r(lds32(lg), lds32(lg + 4), sg), glb = __funnelshift_r(lds32(lg + 32), lds32(lg + 36), sg);
                            const uint32_t hla = __funnelshift_r(lds32(lh), lds32(lh + 4), sh), hlb = __funnelshift_r(lds32(lh + 32), lds32(lh + 36), sh);
                            const uint32_t gh = __funnelshift_r(lds32(qg), lds32(qg + 4), sg), hh = __funnelshift_r(lds32(qh), lds32(qh + 4), sh);
                            const float4 w4g = lds_f4(swg), w4h = lds_f4(swg + 128);
                            const f2 wg[4] = {pack2(w4g.x, w4g.x), pack2(w4g.y, w4g.y), pack2(w4g.z, w4g.z), pack2(w4g.w, w4g.w)};
                            const f2 wh[4] = {pack2(w4h.x, w4h.x), pack2(w4h.y, w4h.y), pack2(w4h.z, w4h.z), pack2(w4h.w, w4h.w)};
                            const uint32_t ag[4] = {(gla & 0x0f0f0f0fu) | ((gh << 4) & 0x30303030u), (glb & 0x0f0f0f0fu) | ((gh << 2) & 0x30303030u),
                                                    ((gla >> 4) & 0x0f0f0f0fu) | (gh & 0x30303030u), ((glb >> 4) & 0x0f0f0f0fu) | ((gh >> 2) & 0x30303030u)};
                            const uint32_t ah[4] = {(hla & 0x0f0f0f0fu) | ((hh << 4) & 0x30303030u), (hlb & 0x0f0f0f0fu) | ((hh << 2) & 0x30303030u),
                                                    ((hla >> 4) & 0x0f0f0f0fu) | (hh & 0x30303030u), ((hlb >> 4) & 0x0f0f0f0fu) | ((hh >> 2) & 0x30303030u)};
#pragma unroll
                            for (int q = 0; q < 4; q++) {
                                int c[4];
                                f2 dxq, tq;
                                mma_k16(c, ag[q], ah[q], b[u][q], kI2FMagicBits, kI2FMagicBits);
                                lds_2f2(ta + 64u * q, dxq, tq);
                                const f2 ntq = tq ^ 0x8000000080000000ull;    // -T: fma(-w, T, acc) == fma(w, -T, acc)
                                ag_ = fma2(wg[q], mul2(dxq, sub2(pack2i(c[0], c[1]), magic2)), ag_);
                                ah_ = fma2(wh[q], mul2(dxq, sub2(pack2i(c[2], c[3]), magic2)), ah_);
                                ag_ = fma2(wg[q], ntq, ag_);
                                ah_ = fma2(wh[q], ntq, ah_);
                            }
                        } else {
                            constexpr int kQs = FMT == FMT_Q5_K ? 48 : 16;
                            const uint32_t e8 = (uint32_t)(8 * (t >> 1) + 16 * (t & 1)), off = (uint32_t)(u * 4 * kSb);
                            const uint2 qg = lds64(base_g + e8 + off + kQs + 32 * jj), qh = lds64(base_h + e8 + off + kQs + 32 * jj);
                            uint32_t lo[4] = {qg.x & 0x0f0f0f0fu, qh.x & 0x0f0f0f0fu, qg.y & 0x0f0f0f0fu, qh.y & 0x0f0f0f0fu};
                            uint32_t hi[4] = {qg.x & 0xf0f0f0f0u, qh.x & 0xf0f0f0f0u, qg.y & 0xf0f0f0f0u, qh.y & 0xf0f0f0f0u};
                            if constexpr (FMT == FMT_Q5_K) {
                                // bits 2j and 2j + 1 of every qh byte are the fifth bits of the two sub-blocks; the high nibbles
                                // go back to plain values (16 * 16 does not fit a byte)
                                const uint2 fg = lds64(base_g + e8 + off + 16), fh = lds64(base_h + e8 + off + 16);
                                const uint32_t f4[4] = {fg.x, fh.x, fg.y, fh.y};
#pragma unroll
                                for (int i = 0; i < 4; i++) {
                                    const uint32_t x = f4[i] >> (2 * jj);
                                    lo[i] |= (x << 4) & 0x10101010u;
                                    hi[i] = (hi[i] >> 4) | ((x << 3) & 0x10101010u);
                                }
                            }
                            f2 dx0, s0, dx1, s1;
                            int c[4], e[4];
                            mma_k32<false>(c, lo[0], lo[1], lo[2], lo[3], b[u][0], b[u][1], kI2FMagicBits, kI2FMagicBits);
                            mma_k32<false>(e, hi[0], hi[1], hi[2], hi[3], b[u][2], b[u][3], kI2FMagicBits, kI2FMagicBits);
                            const float4 wg = lds_f4(swg), wh = lds_f4(swg + 128);
                            lds_2f2(ta, dx0, s0);
                            lds_2f2(ta + 64, dx1, s1);
                            const f2 wsg0 = pack2(wg.x, wg.x), wog0 = pack2(wg.y, wg.y), wsg1 = pack2(wg.z, wg.z), wog1 = pack2(wg.w, wg.w);
                            const f2 wsh0 = pack2(wh.x, wh.x), woh0 = pack2(wh.y, wh.y), wsh1 = pack2(wh.z, wh.z), woh1 = pack2(wh.w, wh.w);
                            ag_ = fma2(wsg0, mul2(dx0, sub2(pack2i(c[0], c[1]), magic2)), ag_);
                            ah_ = fma2(wsh0, mul2(dx0, sub2(pack2i(c[2], c[3]), magic2)), ah_);
                            ag_ = fma2(wog0, s0, ag_);
                            ah_ = fma2(woh0, s0, ah_);
                            ag_ = fma2(wsg1, mul2(dx1, sub2(pack2i(e[0], e[1]), magic2)), ag_);
                            ah_ = fma2(wsh1, mul2(dx1, sub2(pack2i(e[2], e[3]), magic2)), ah_);
                            ag_ = fma2(wog1, s1, ag_);
                            ah_ = fma2(woh1, s1, ah_);
                        }
                    }
                }
            }
            };
            if (nu == 5) multiply(std::integral_constant<int, 5>{});
            else if (nu == 4) multiply(std::integral_constant<int, 4>{});
            else multiply(std::integral_constant<int, 0>{});
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(empty_bar(slot)) : "memory");
            if (++slot == S) {
                slot = 0;
                par ^= 1u;
            }
            if (pass < p.npass - 1) {
                *reinterpret_cast<ulonglong2 *>(keep + (swap ? kPart / 2 : 0)) = make_ulonglong2(acc[0][0], acc[0][1]);
                *reinterpret_cast<ulonglong2 *>(keep + (swap ? 0 : kPart / 2)) = make_ulonglong2(acc[1][0], acc[1][1]);
            } else {
                const int pb = done & 1;
                ok = mbar_wait(pempty_bar(pb), ((uint32_t)(done >> 1) & 1u) ^ 1u, p.status, (12u << 24) | 0x100u | (uint32_t)pb);
                if (!__all_sync(0xffffffffu, ok)) return;
                // the butterfly's first step: lane w + lane (w + 16)
                *reinterpret_cast<ulonglong2 *>(s_part + ((size_t)pb * kConsumers + warp) * kPart + 4 * lane) =
                    make_ulonglong2(add2(acc[0][0], acc[1][0]), add2(acc[0][1], acc[1][1]));
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(pfull_bar(pb)) : "memory");
                done++;
            }
        }
    }
}

struct KmmaPlan {
    int npass = 0, blk_rg = 0, pitch = 0, stages = 0, grid = 0;
    size_t smem = 0;
};

// The fewest passes over K whose stages fit two deep beside the tables and, with more than one, the accumulators of four row
// groups (or as many as a CTA has).  Deeper rings at the price of another pass were slower: q6_k 5120 x 17408 43 us in six passes
// of two stages, 48 in ones of three.
KmmaPlan plan_kmma(tpb_handle_t h, int fmt, int64_t rows, int64_t cols) {
    const int n_sb = (int)(cols / 256), n_grp4 = (n_sb + 3) / 4;
    long long grid = (rows + 3) / 4;      // few rows: row groups of down to four keep more SMs streaming
    if (grid > h->sm_count) grid = h->sm_count;
    const int n_rg = (int)(((rows + grid - 1) / grid + kRows - 1) / kRows);
    const size_t limit = (size_t)h->smem_optin - 1024;
    const size_t fixed = (size_t)kConsumers * (NU * tab_bytes(fmt) + kSwBytes) + (size_t)2 * kConsumers * kPart * 4 + 160;
    KmmaPlan pl;
    for (int npass = (n_grp4 + NU - 1) / NU; npass <= n_grp4; npass++) {
        const int grp = (n_grp4 + npass - 1) / npass;                    // groups of the largest pass
        const int sbs = 4 * grp < n_sb ? 4 * grp : n_sb;
        // q6_k: up to 15 bytes of misalignment, the rounded copy and a word read past the last field
        int pitch = sbs * sb_bytes(fmt) + (fmt == FMT_Q6_K ? 36 : 0);
        pitch = (pitch + 79) / 128 * 128 + 48;
        const int blk = npass == 1 ? n_rg : n_rg < 4 ? n_rg : 4;
        const size_t acc = npass == 1 ? 0 : (size_t)blk * kConsumers * 2 * kPart * 4;
        if (fixed + acc >= limit) return pl;
        int stages = (int)((limit - fixed - acc) / ((size_t)kRows * pitch));
        if (stages > 8) stages = 8;
        if (stages < 2) continue;
        pl.npass = npass;
        pl.blk_rg = blk;
        pl.pitch = pitch;
        pl.stages = stages;
        pl.grid = (int)grid;
        pl.smem = fixed + acc + (size_t)stages * kRows * pitch;
        return pl;
    }
    return pl;
}

template <int FMT>
int launch_kmma(tpb_handle_t h, cudaStream_t st, const KmmaParams &p, const KmmaPlan &pl) {
    auto kern = kquant_gemv_mma_kernel<FMT>;
    static tpb_per_device_once smem_set;
    TPB_CUDA(h, tpb_set_max_smem_once(h, kern, h->smem_optin, smem_set));
    TPB_CUDA(h, tpb_launch_pdl(kern, dim3((unsigned)pl.grid), dim3(kThreads), pl.smem, st, p));
    return TPB_OK;
}

}  // namespace

// Whether the kernel takes such a weight.
bool tpb_kquant_mma_fits(tpb_handle_t h, int fmt, int64_t rows, int64_t cols) { return cols % 256 == 0 && plan_kmma(h, fmt, rows, cols).npass != 0; }

int tpb_launch_kquant_mma(tpb_handle_t h, cudaStream_t st, int fmt, float *y, const uint8_t *w, float scale, int64_t rows,
                          int64_t cols, const float *xd, const int8_t *xq, int m) {
    const KmmaPlan pl = plan_kmma(h, fmt, rows, cols);
    if (pl.npass == 0) return tpb_fail(h, TPB_ERR_INVALID_ARG, "gguf_gemv: %lld columns do not fit the register-resident kernel", (long long)cols);
    KmmaParams p;
    p.y = y;
    p.w = w;
    p.xd = xd;
    p.xq = xq;
    p.scale = scale;
    p.rows = (int)rows;
    p.cols = (int)cols;
    p.nblk = (int)(cols / 32);
    p.m = m;
    p.npass = pl.npass;
    p.blk_rg = pl.blk_rg;
    p.pitch = pl.pitch;
    p.stages = pl.stages;
    p.row_bytes = (uint32_t)(cols / 256) * (uint32_t)sb_bytes(fmt);
    p.status = h->d_status;
    switch (fmt) {
        case FMT_Q4_0: return launch_kmma<FMT_Q4_0>(h, st, p, pl);
        case FMT_Q4_K: return launch_kmma<FMT_Q4_K>(h, st, p, pl);
        case FMT_Q5_K: return launch_kmma<FMT_Q5_K>(h, st, p, pl);
        case FMT_Q6_K: return launch_kmma<FMT_Q6_K>(h, st, p, pl);
        default: return launch_kmma<FMT_IQ4_NL>(h, st, p, pl);
    }
}
