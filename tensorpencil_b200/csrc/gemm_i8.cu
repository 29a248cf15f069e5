// ConvRot int8 GEMM with fused dequant epilogue for sm_100a.
//
//   y[i][j] = (float(sum_k q[i][k] * w[j][k]) * act_scale[i]) * w_scale[j]
//
// Both operands are K-major (q is [m][k], w is [n][k]) so neither is transposed.
// One persistent CTA per SM walks output tiles of 128 x BN:
//   warp 0      : TMA producer -- 128-byte-swizzled tiles of q and w, K block of
//                 128 bytes per pipeline stage, completion on an mbarrier;
//   warp 1      : allocates TMEM and issues tcgen05.mma.kind::i8 (M=128, N=BN = 64 .. 256,
//                 K=32) from one thread; int32 accumulators live in TMEM, two
//                 buffers so the epilogue of tile t overlaps the main loop of t+1;
//   warps 2..5  : epilogue -- tcgen05.ld the accumulator rows (the load of the
//                 next 32 columns is in flight while the current ones are
//                 processed), apply the two scales, convert, stage the 32-row x
//                 128-byte piece in shared memory in the 128-byte swizzle
//                 pattern and hand it to a TMA store, so global memory sees
//                 whole 128-byte lines; two staging buffers per warp.
// Every wait on an mbarrier is bounded: on expiry the kernel records a status
// word, every role leaves its loop, TMEM is released and the kernel returns.
// No TMA load here uses cluster multicast.
#include <cstdlib>

#include "gemm_common.cuh"

int tpb_launch_gemm2_group(tpb_handle_t h, cudaStream_t st, const tpb_gemm::GemmParams &p, int y_dtype, const int8_t *q,
                           int count, const void *const *w8, const float *const *w_scale, void *const *y);
int tpb_launch_gemm2_silu_pair(tpb_handle_t h, cudaStream_t st, const tpb_gemm::GemmParams &p, int y_dtype,
                               const int8_t *q, const void *w_gate, const void *w_up);
int tpb_launch_gemm2(tpb_handle_t h, cudaStream_t st, const tpb_gemm::GemmParams &p, int y_dtype,
                     const int8_t *q, const void *w8, bool b_unsigned);
int tpb_launch_gemm_splitk(tpb_handle_t h, cudaStream_t st, const tpb_gemm::GemmParams &p, int y_dtype, const int8_t *q, const void *w8,
                           int bn, int split);
int tpb_launch_gemm_w4(tpb_handle_t h, cudaStream_t st, const tpb_gemm::GemmParams &p, int y_dtype,
                        const int8_t *q, const void *w4);

namespace {

using namespace tpb_gemm;

// ---- the kernel ---------------------------------------------------------------

template <int BN, int OUT, int PEERS>
__global__ void __launch_bounds__(kThreads, 1)
convrot_gemm_kernel(const __grid_constant__ CUtensorMap tma_a,
                    const __grid_constant__ CUtensorMap tma_b,
                    const __grid_constant__ CUtensorMap tma_y, const GemmParams p,
                    const int b_unsigned) {
    using Cfg = TileCfg<BN>;
    constexpr int S = Cfg::kStages;

    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    // layout: [S x (A tile | B tile)] [epilogue staging] [barriers] [tmem slot] [abort flag]
    const uint32_t stg_base = smem_base + S * Cfg::kStageBytes;
    const uint32_t bars = stg_base + Cfg::kStagingBytes;
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (S + s); };
    auto tfull_bar = [&](int a) { return bars + 8u * (2 * S + a); };
    auto tempty_bar = [&](int a) { return bars + 8u * (2 * S + 2 + a); };
    uint8_t *tail = smem_gen + S * Cfg::kStageBytes + Cfg::kStagingBytes + 8 * (2 * S + 4);
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(tail);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tail + 8);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    const int m_tiles = (p.m + BM - 1) / BM;
    const int n_tiles = (p.n + BN - 1) / BN;
    const int num_tiles = m_tiles * n_tiles;
    const int k_blocks = p.k / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), 4);  // one arrival per epilogue warp
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32((const void *)tmem_slot)),
                     "r"(Cfg::kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // set-up above overlaps the previous kernel's tail; global memory only after this
    tpb_grid_dep_launch();
    tpb_grid_dep_wait();

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x) {
                const int m0 = (tile % m_tiles) * BM;
                const int n0 = (tile / m_tiles) * BN;
                for (int kb = 0; kb < k_blocks; kb++, it++) {
                    const int s = it % S;
                    const uint32_t ph = (it / S) & 1u;
                    ok = mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, p.status, (1u << 24) | s, true);
                    if (!ok) break;
                    mbar_arrive_expect_tx(full_bar(s), Cfg::kStageBytes);
                    const uint32_t a_dst = smem_base + s * Cfg::kStageBytes;
                    tma_load_2d(a_dst, &tma_a, full_bar(s), kb * BK, m0);
                    tma_load_2d(a_dst + Cfg::kStageBytesA, &tma_b, full_bar(s), kb * BK, n0);
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            const uint32_t idesc = make_idesc_i8<BN>(b_unsigned != 0);
            uint32_t it = 0, t_it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x, t_it++) {
                const int acc = t_it & 1;
                const uint32_t acc_ph = (t_it >> 1) & 1u;
                ok = mbar_wait(tempty_bar(acc), acc_ph ^ 1u, abort_flag, p.status, (2u << 24) | 0x100u | acc);
                if (!ok) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN);
                for (int kb = 0; kb < k_blocks; kb++, it++) {
                    const int s = it % S;
                    const uint32_t ph = (it / S) & 1u;
                    ok = mbar_wait(full_bar(s), ph, abort_flag, p.status, (2u << 24) | s);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t a_addr = smem_base + s * Cfg::kStageBytes;
                    const uint64_t a_desc = make_kmajor_sw128_desc(a_addr);
                    const uint64_t b_desc = make_kmajor_sw128_desc(a_addr + Cfg::kStageBytesA);
#pragma unroll
                    for (int kk = 0; kk < BK / UMMA_K; kk++) {
                        // advancing 32 bytes inside the 128-byte swizzle row = +2 in the
                        // (address >> 4) field of the descriptor
                        tc_mma_i8(d_tmem, a_desc + 2u * kk, b_desc + 2u * kk, idesc,
                                  (kb > 0 || kk > 0) ? 1u : 0u);
                    }
                    tc_commit(empty_bar(s));  // stage reusable once these MMAs have read it
                }
                if (ok) tc_commit(tfull_bar(acc));  // accumulator complete
            }
        }
    } else {
        // ---------------- epilogue ----------------
        const int quarter = warp & 3;  // TMEM lane quarter this warp may access
        // two 4 KB staging buffers per warp (BN = 192: one), each 32 rows x 128 bytes, 1024-byte aligned
        const uint32_t stg = stg_base + (uint32_t)(warp - 2) * (uint32_t)Cfg::kStagingPerWarp;
        const uint32_t my_row_off = (uint32_t)lane * 128u;
        const uint32_t sw = (uint32_t)(lane & 7);  // 128-byte swizzle: 16-byte piece j of row r sits at j ^ (r & 7)
        uint32_t n_store = 0;                      // stores issued by this warp (selects the staging buffer)
        uint32_t t_it = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x, t_it++) {
            const int m0 = (tile % m_tiles) * BM;
            const int n0 = (tile / m_tiles) * BN;
            const int acc = t_it & 1;
            const uint32_t acc_ph = (t_it >> 1) & 1u;
            ok = mbar_wait(tfull_bar(acc), acc_ph, abort_flag, p.status, (3u << 24) | acc, true);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const int row0 = m0 + quarter * 32;
            const int row = row0 + lane;
            const bool row_ok = row < p.m;
            float as = 0.0f;
            int corr = 0;
            if (OUT != OUT_S32 && row_ok) as = __ldcg(p.act_scale + row);
            if (p.act_sum != nullptr && row_ok) corr = 8 * __ldcg(p.act_sum + row);
            const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN);

            epilogue_tile<BN, OUT, PEERS, false, Cfg::kOneStaging>(t_row, p, &tma_y, stg, my_row_off, sw, n_store, row0, n0, as, corr, lane);
            // all of this warp's TMEM reads are complete: hand the buffer back
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty_bar(acc));
        }
        // staging memory must outlive the stores that read it
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
    }

    // ---------------- teardown ----------------
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        // A role gave up.  Give copies and MMAs still in flight time to land
        // before shared memory and TMEM are released.
        for (int i = 0; i < 200; i++) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                     "r"(Cfg::kTmemCols)
                     : "memory");
    }
}

// ---- host side ------------------------------------------------------------------

template <int BN, int OUT, int PEERS>
int launch_cfg_p(tpb_handle_t h, cudaStream_t st, const GemmParams &p, const int8_t *q, const void *w8,
               bool b_unsigned) {
    using Cfg = TileCfg<BN>;
    CUtensorMap ma, mb, my;
    int rc = make_kmajor_map(h, &ma, q, p.m, p.k, BM);
    if (rc != TPB_OK) return rc;
    rc = make_kmajor_map(h, &mb, w8, p.n, p.k, BN);
    if (rc != TPB_OK) return rc;
    rc = make_out_map<OUT>(h, &my, p);
    if (rc != TPB_OK) return rc;
    auto kern = convrot_gemm_kernel<BN, OUT, PEERS>;
    static tpb_per_device_once smem_set;   // per instantiation
    TPB_CUDA(h, tpb_set_max_smem_once(h, kern, Cfg::kSmemBytes, smem_set));
    const int m_tiles = (p.m + BM - 1) / BM, n_tiles = (p.n + BN - 1) / BN;
    const int tiles = m_tiles * n_tiles;
    const int grid = tiles < h->sm_count ? tiles : h->sm_count;
    TPB_CUDA(h, tpb_launch_pdl(kern, dim3(grid), dim3(kThreads), Cfg::kSmemBytes, st, ma, mb, my, p, b_unsigned ? 1 : 0));
    return TPB_OK;
}

template <int BN, int OUT>
int launch_cfg(tpb_handle_t h, cudaStream_t st, const GemmParams &p, const int8_t *q, const void *w8,
               bool b_unsigned) {
    if (p.gate != nullptr) return launch_cfg_p<BN, OUT_F32, 3>(h, st, p, q, w8, b_unsigned);
    if constexpr (BN != 192) {   // pick_tile_peers
        if (p.mc_y != nullptr) return launch_cfg_p<BN, OUT, 2>(h, st, p, q, w8, b_unsigned);
        if (p.n_peers > 0) return launch_cfg_p<BN, OUT, 1>(h, st, p, q, w8, b_unsigned);
    }
    return launch_cfg_p<BN, OUT, 0>(h, st, p, q, w8, b_unsigned);
}

// Which tile takes a problem: the one whose waves of tiles cost least.  A persistent CTA (or CTA pair) walks whole tiles, ceil(tiles /
// SMs) rounds of them, with the epilogue of one tile beside the K blocks of the next: launch and pipeline fill, the first round's K blocks,
// for every further round its K blocks or the epilogue, whichever takes longer, and the last epilogue.  Fitted to 241 shapes (m 130 ..
// 4608, n 1024 .. 12288, k 256 .. 12288) times five tiles times three epilogues, rms error 6-8 % (us: fixed, per K block of 128, epilogue to
// f32 / to bf16 / gated residual):
//   128 x 64    1.9   0.295   1.3  1.0   2.5   (bound by shared-memory traffic: A is staged for 64 columns only)
//   128 x 128   1.7   0.307   2.4  1.8   5.4
//   128 x 192   1.9   0.312   3.9  2.7   8.1
//   128 x 256   1.7   0.395   4.9  3.9  10.6
//   256 x 256   2.0   0.338   5.3  4.5   9.3   on an SM pair
// The choice is within 0.5 % of the best tile on average.  E.g. m 1111, n 3072, k 12288: 216 tiles of 128 x 128 are two rounds, 60 us; 144 of
// 128 x 192 are one, 35 us.  m 777, n 2048, k 4096: two rounds of 128 x 64 23 us, one of 128 x 128 14.7.  m 2048, n 3072, k 12288: 96 pair tiles
// on 74 pairs 69 us, 176 of 128 x 192 64 us.  m 3000, n 1536, k 1024: 72 pair tiles 10.7 us, two rounds of 128 x 128 9.8 (with the epilogue left out
// of the rounds the pair looked cheaper).  The pair keeps a problem unless another tile is 8 % better (gated: 4 %): under the power cap,
// which a long GEMM meets, its fewer bytes staged per product count for more than the bursts above show.
enum Tile { S64, S128, S192, S256, P256 };
enum Epilogue { EPI_F32, EPI_BF16, EPI_GATED };
double tile_us(int sms, Tile t, Epilogue epi, int64_t m, int64_t n, int64_t k, int count) {
    static const struct { int bm, bn, sms; double fixed, per_block, epilogue[3]; } kCost[] = {
        {128, 64, 1, 1.9, 0.295, {1.3, 1.0, 2.5}}, {128, 128, 1, 1.7, 0.307, {2.4, 1.8, 5.4}}, {128, 192, 1, 1.9, 0.312, {3.9, 2.7, 8.1}},
        {128, 256, 1, 1.7, 0.395, {4.9, 3.9, 10.6}}, {256, 256, 2, 2.0, 0.338, {5.3, 4.5, 9.3}}};
    const auto &c = kCost[t];
    const int64_t tiles = (m + c.bm - 1) / c.bm * ((n + c.bn - 1) / c.bn) * count;
    const int64_t slots = sms / c.sms > 0 ? sms / c.sms : 1;
    const double blocks = (double)(k / BK) * c.per_block, e = c.epilogue[epi];
    return c.fixed + blocks + (double)((tiles + slots - 1) / slots - 1) * (blocks > e ? blocks : e) + e;
}
Tile pick_tile(tpb_handle_t h, Epilogue epi, int64_t m, int64_t n, int64_t k, double *us = nullptr) {
    // A gated residual larger than half of L2 or so: its reads and writes bound the launch, and the pair with its eight epilogue warps
    // has most of them in flight (4608 x 3072, k 3072: pair 43.6 us, 128 x 192 52.7; 3000 x 8192, k 512: 63.7 against 69-93).
    if (epi == EPI_GATED && m * n >= 14000000 && !h->opt_gemm_one_cta) return P256;
    Tile best = S64;
    double t_best = 0.0;
    for (int t = S64; t <= P256; t++) {
        if (t == P256 && h->opt_gemm_one_cta) break;
        const double raw = tile_us(h->sm_count, (Tile)t, epi, m, n, k, 1);
        const double v = t == P256 ? raw * (epi == EPI_GATED ? 0.96 : 0.92) : raw;
        if (t == S64 || v < t_best) {
            best = (Tile)t;
            t_best = v;
            if (us) *us = raw;
        }
    }
    return best;
}
// Whether the CTAs of a cluster share a tile's K (gemm_splitk.cu), and how: for problems whose tiles leave SMs idle and whose K is a long chain.
// One round of clusters only, as many as the device holds at once; the cost of a choice is linear in the K blocks of a part, the rows whose
// parts are sent and added, and the bytes that all SMs load (us, fitted to 128 shapes x 18 choices, rms error 6-8 %).  us, one
// chain / split: m 16, n 1024, k 12288 29.4 / 8.3; m 64, n 3072, k 6144 16.8 / 8.8; m 256, n 1024, k 3072 10.1 / 6.3; m 256, n = k = 3072 10.5 / 9.0;
// m 297, n 3072, k 12288 30.6 / 22.2.  Over 384 shapes and epilogues with m 16 .. 1111 the choice is 1.28 x as fast as
// one chain on average and 2 % slower at worst, over 200 others with m 1 .. 1400 4 % at worst (m 642, n 1424, k 512 gated 6.8 / 7.1), at k 256 5 % (m 204, n 912 to s32 3.1 / 3.3).  Several rounds of clusters lost everywhere (m 512, n 5008, k 3072: 13.9 / 25 and more).
struct Split { int bn = 0, parts = 1; double us = 0.0; };
Split pick_split(tpb_handle_t h, int64_t m, int64_t n, int64_t k, double one_cta_us) {
    static const struct { int bn; double fixed, per_block, rows, rows_part, load; } kCost[] = {
        {64, 2.84, 0.260, 1.51, -2.13, 0.112}, {128, 3.10, 0.345, 2.08, -2.10, 0.080}, {192, 3.49, 0.352, 2.85, -1.90, 0.265}};
    Split best;
    double t_best = 0.96 * one_cta_us;
    const int64_t blocks = k / BK;
    if (h->opt_gemm_one_cta || h->opt_gemm_split_bn == 0) return best;
    if (h->opt_gemm_split_bn > 0) {
        const int64_t tiles = (m + BM - 1) / BM * ((n + h->opt_gemm_split_bn - 1) / h->opt_gemm_split_bn);
        if (h->opt_gemm_split_parts <= blocks && tiles <= h->max_clusters[h->opt_gemm_split_parts]) {
            best.bn = h->opt_gemm_split_bn;
            best.parts = h->opt_gemm_split_parts;
            best.us = t_best;
        }
        return best;
    }
    const double rows = (double)(m < BM ? m : BM) / BM;
    // Parts of a single K block of full tiles with few columns: there is next to no chain, and the one-chain kernel's epilogue stores less than its cost
    // says (m 193, n 32, k 256 3.0 one chain / 3.35 split; but m 5, n 16 2.8 / 2.3, m 185, n 1360 gated 4.9 / 3.85).
    if (blocks < 4 && m > BM && n <= 96) return best;
    for (const auto &c : kCost) {
        const int64_t tiles = (m + BM - 1) / BM * ((n + c.bn - 1) / c.bn);
        for (int parts = 2; parts <= kMaxSplit && parts <= blocks; parts++) {
            if (tiles > h->max_clusters[parts]) break;
            const double b = (double)((blocks + parts - 1) / parts);
            const double us = c.fixed + c.per_block * b + c.rows * rows + c.rows_part * rows / parts + c.load * b * (double)(tiles * parts) / h->sm_count;
            if (us < t_best) {
                best.bn = c.bn;
                best.parts = parts;
                best.us = t_best = us;
            }
        }
    }
    return best;
}
// The fused all-gather's epilogue also writes every other GPU's copy of the output, which the costs above do not hold:
// there the widest tile that still gives every SM (pair) work.
Tile pick_tile_peers(tpb_handle_t h, int64_t m, int64_t n) {
    auto tiles = [&](int bm, int bn) { return (m + bm - 1) / bm * ((n + bn - 1) / bn); };
    if (!h->opt_gemm_one_cta && tiles(256, 256) >= h->sm_count / 2) return P256;
    return tiles(128, 256) >= h->sm_count ? S256 : tiles(128, 128) >= h->sm_count ? S128 : S64;
}

template <int OUT>
int launch_out(tpb_handle_t h, cudaStream_t st, const GemmParams &p, const int8_t *q, const void *w8,
               bool b_unsigned, Tile tile) {
    switch (tile) {
        case S256: return launch_cfg<256, OUT>(h, st, p, q, w8, b_unsigned);
        case S192: return launch_cfg<192, OUT>(h, st, p, q, w8, b_unsigned);
        case S128: return launch_cfg<128, OUT>(h, st, p, q, w8, b_unsigned);
        default: return launch_cfg<64, OUT>(h, st, p, q, w8, b_unsigned);
    }
}

}  // namespace

int tpb_w4_scratch(tpb_handle_t h, int64_t n, int64_t k, int8_t **out) {
    const size_t need = (size_t)n * (size_t)k;
    if (h->w4_scratch_bytes < need)
        return tpb_fail(h, TPB_ERR_STATE,
                        "int4 weight of %lld x %lld needs %zu bytes of expansion scratch, %zu reserved: call "
                        "tpb_convrot_w4_reserve(h, n, k) once, outside the stream-ordered path",
                        (long long)n, (long long)k, need, h->w4_scratch_bytes);
    *out = h->w4_scratch;
    return TPB_OK;
}

int tpb_launch_gemm(tpb_handle_t h, cudaStream_t st, void *y, int y_dtype, int64_t ldy,
                    const int8_t *q, const float *act_scale, const int32_t *act_sum, const void *w,
                    int w_bits, const float *w_scale, int64_t m, int64_t n, int64_t k,
                    void *const *peer_y, int n_peers, void *mc_y, const float *gate) {
    GemmParams p;
    p.mc_y = mc_y;
    p.gate = gate;
    p.ablate = h->opt_gemm_ablate;
    p.n_peers = n_peers;
    for (int i = 0; i < kMaxPeers; i++) p.peer_y[i] = i < n_peers ? peer_y[i] : nullptr;
    p.y = y;
    p.ldy = ldy;
    p.act_scale = act_scale;
    p.w_scale = w_scale;
    p.act_sum = nullptr;
    p.m = (int)m;
    p.n = (int)n;
    p.k = (int)k;
    p.status = h->d_status;
    const void *w8 = w;
    if (w_bits == 4 && n_peers == 0 && mc_y == nullptr && gate == nullptr && h->opt_w4_fused &&
        ((m + 127) / 128) * ((n + 255) / 256) >= h->sm_count) {
        // opt-in: the packed weight is unpacked inside the GEMM (one-CTA kernel)
        p.act_sum = act_sum;
        return tpb_launch_gemm_w4(h, st, p, y_dtype, q, w);
    }
    if (w_bits == 4) {
        int8_t *buf = nullptr;
        int rc = tpb_w4_scratch(h, n, k, &buf);
        if (rc != TPB_OK) return rc;
        rc = tpb_launch_w4_expand(h, st, w, n, k, buf);
        if (rc != TPB_OK) return rc;
        w8 = buf;
    }
    // TPB_GEMM_ONE_CTA=1 keeps the one-CTA kernel for comparisons, TPB_GEMM_SPLIT=0 or "columns,parts" whether and how K is split.
    Tile tile;
    if (n_peers > 0 || mc_y != nullptr) {
        tile = pick_tile_peers(h, m, n);
    } else {
        double us = 0.0;
        tile = pick_tile(h, gate ? EPI_GATED : y_dtype == TPB_BF16 ? EPI_BF16 : EPI_F32, m, n, k, &us);
        const Split split = pick_split(h, m, n, k, us);   // (one part under TPB_GEMM_ONE_CTA)
        if (split.parts > 1) return tpb_launch_gemm_splitk(h, st, p, y_dtype, q, w8, split.bn, split.parts);
    }
    if (tile == P256) return tpb_launch_gemm2(h, st, p, y_dtype, q, w8, false);
    switch (y_dtype) {
        case TPB_F32: return launch_out<OUT_F32>(h, st, p, q, w8, false, tile);
        case TPB_BF16: return launch_out<OUT_BF16>(h, st, p, q, w8, false, tile);
        case TPB_S32: return launch_out<OUT_S32>(h, st, p, q, w8, false, tile);
    }
    return tpb_fail(h, TPB_ERR_INVALID_ARG, "gemm: unsupported y_dtype %d", y_dtype);
}

// y = silu(gate projection) * (up projection): both weights multiplied in one launch of the two-CTA
// kernel (each CTA of a pair brings in one weight's half of the tile), combined in its epilogue.
int tpb_launch_gemm_silu_pair(tpb_handle_t h, cudaStream_t st, void *y, int y_dtype, int64_t ldy, const int8_t *q,
                              const float *act_scale, const void *w_gate, const float *w_gate_scale, const void *w_up,
                              const float *w_up_scale, int w_bits, int64_t m, int64_t n, int64_t k) {
    GemmParams p;
    p.mc_y = nullptr;
    p.gate = nullptr;
    p.ablate = 0;
    p.n_peers = 0;
    for (int i = 0; i < kMaxPeers; i++) p.peer_y[i] = nullptr;
    p.y = y;
    p.ldy = ldy;
    p.act_scale = act_scale;
    p.w_scale = w_gate_scale;
    p.w_scale2 = w_up_scale;
    p.act_sum = nullptr;
    p.m = (int)m;
    p.n = (int)n;
    p.k = (int)k;
    p.status = h->d_status;
    const void *g8 = w_gate, *u8 = w_up;
    if (w_bits == 4) {
        // both weights widened into the reserved scratch, one after the other
        int8_t *buf = nullptr;
        int rc = tpb_w4_scratch(h, 2 * n, k, &buf);
        if (rc != TPB_OK) return rc;
        rc = tpb_launch_w4_expand(h, st, w_gate, n, k, buf);
        if (rc != TPB_OK) return rc;
        rc = tpb_launch_w4_expand(h, st, w_up, n, k, buf + (size_t)n * (size_t)k);
        if (rc != TPB_OK) return rc;
        g8 = buf;
        u8 = buf + (size_t)n * (size_t)k;
    }
    return tpb_launch_gemm2_silu_pair(h, st, p, y_dtype, q, g8, u8);
}

// Up to four weights of one shape times the same activations in one launch of the two-CTA kernel (the q, k, v and
// gate projections of a DiT block): their tiles follow one another in its persistent loop, so the pipeline fills
// and drains once instead of once per weight, and the last round is shared by all of them.  One by one where a tile of
// the one-CTA kernel fits a single weight so much better that it pays: two weights of m 2048, n 12288, k 512 to bf16 46 us one by one,
// 54 together, of m 256, n 3072, k 256 7.3 / 8.0; but four of m 256, n = k = 3072 41 / 17, four of m 1111, n 3072, k 12288 143 / 141.
// A weight whose K is split over a cluster is a shorter single call, but a split launch right behind another takes up to a fifth more than alone, so
// it has to be 15 % better than the group: us, together / one by one with K split: two of m 49, n 384, k 8960 27.3 / 11.8, three of m 2, n 704, k 7936 25.8 /
// 17.1; but four of m 3, n 960, k 4608 18.1 / 23.9.  Over 114 groups of m 1 .. 700 the choice is 0.5 % off the better route on average (8.8 without).
int tpb_launch_gemm_group(tpb_handle_t h, cudaStream_t st, int count, void *const *y, int y_dtype, int64_t ldy,
                          const int8_t *q, const float *act_scale, const int32_t *act_sum, const void *const *w,
                          const float *const *w_scale, int w_bits, int64_t m, int64_t n, int64_t k) {
    const Epilogue epi = y_dtype == TPB_BF16 ? EPI_BF16 : EPI_F32;
    double one_us = 0.0;
    pick_tile(h, epi, m, n, k, &one_us);
    const Split split = pick_split(h, m, n, k, one_us);
    // A reservation that covers one int4 weight only is enough for small problems, as it was when they always ran one by one.
    const bool small = (m + 255) / 256 * ((n + 255) / 256) < h->sm_count / 2;
    const bool scratch_for_one = w_bits == 4 && small && h->w4_scratch_bytes < (size_t)count * (size_t)n * (size_t)k;
    // A larger one needs every weight reserved, whichever route is the faster.
    int8_t *all_weights = nullptr;
    if (w_bits == 4 && !small && !h->opt_gemm_one_cta) {
        const int rc = tpb_w4_scratch(h, (int64_t)count * n, k, &all_weights);
        if (rc != TPB_OK) return rc;
    }
    // the pair's bonus where it holds (pick_tile): in a launch long enough to meet the power cap
    const double together_us = (small ? 1.0 : 0.96) * tile_us(h->sm_count, P256, epi, m, n, k, count);
    if (h->opt_gemm_one_cta || scratch_for_one || together_us > count * one_us || (split.parts > 1 && 0.85 * together_us > count * split.us)) {
        for (int g = 0; g < count; g++) {
            const int rc = tpb_launch_gemm(h, st, y[g], y_dtype, ldy, q, act_scale, act_sum, w[g], w_bits, w_scale[g], m, n, k,
                                           nullptr, 0, nullptr, nullptr);
            if (rc != TPB_OK) return rc;
        }
        return TPB_OK;
    }
    GemmParams p;
    p.mc_y = nullptr;
    p.gate = nullptr;
    p.ablate = 0;
    p.n_peers = 0;
    for (int i = 0; i < kMaxPeers; i++) p.peer_y[i] = nullptr;
    p.y = y[0];
    p.ldy = ldy;
    p.act_scale = act_scale;
    p.w_scale = w_scale[0];
    p.act_sum = nullptr;
    p.m = (int)m;
    p.n = (int)n;
    p.k = (int)k;
    p.status = h->d_status;
    const void *w8[4] = {nullptr, nullptr, nullptr, nullptr};
    for (int g = 0; g < count; g++) w8[g] = w[g];
    if (w_bits == 4) {
        // every weight widened into the reserved scratch, one after the other
        int8_t *buf = nullptr;
        int rc = tpb_w4_scratch(h, (int64_t)count * n, k, &buf);
        if (rc != TPB_OK) return rc;
        for (int g = 0; g < count; g++) {
            int8_t *dst = buf + (size_t)g * (size_t)n * (size_t)k;
            rc = tpb_launch_w4_expand(h, st, w[g], n, k, dst);
            if (rc != TPB_OK) return rc;
            w8[g] = dst;
        }
    }
    return tpb_launch_gemm2_group(h, st, p, y_dtype, q, count, w8, w_scale, y);
}
