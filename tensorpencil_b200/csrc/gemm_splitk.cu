// ConvRot int8 GEMM with K split over a cluster, for problems with too few tiles to fill the SMs.
//
// A tile's K loop is a serial chain that one SM can feed at no more than ~64 bytes per clock from L2 (a K block of a 128 x 128
// tile: 32 KB, 0.3 us), so a problem of fewer tiles than SMs takes one tile's time however many SMs are idle.  Here the C CTAs of a cluster
// take one tile and a C-th of its K blocks each:
//   warp 0     : TMA producer, warp 1: tcgen05.mma issuer, as in convrot_gemm_kernel, over this CTA's K blocks;
//   warps 2..9 : read the partial accumulators out of tensor memory into shared memory, one row per lane, and send every
//                other CTA of the cluster the rows that it finishes (cp.async.bulk from shared memory to its shared memory, completion on
//                its mbarrier: whole contiguous pieces, no stores of single words through the cluster's network);
//                then add the C parts of the rows that this CTA finishes -- int32, so the order changes no bit -- dequantise and
//                store them, a warp to whole rows of the tile.
// A tile's rows, as far as the problem has them, are split evenly over the cluster, so the last step has the whole cluster's SMs too.
// What bounds it (cycle stamps, m 256, n = k = 3072 as 128 x 128 tiles on 48 pairs, 1.9 GHz): 1500 cycles until the first load is asked for,
// 7200 for twelve K blocks (the first load's latency, then 600 a block: L2 to SM), and, with four warps for it, 1150 to stage and send the parts, 1350 until the
// peer's are there, 3350 for sums and stores; eight warps took the launch from 9.5 to 9.0 us.  One barrier.cluster.sync at each end cost 500 and
// 1300 more; parts padded to 144 bytes a row instead of swizzled left no room for 192 columns.
// Every wait is bounded, and the cluster barrier at the end keeps a CTA's shared memory alive until all its copies have arrived.  No
// load or copy here uses cluster multicast.
#include "gemm_common.cuh"

namespace {

using namespace tpb_gemm;

// Eight warps for the sums, two to a quarter of tensor memory: with four, one to a scheduler, their straight-line code ran at three to four cycles an
// instruction (128 x 128, two parts: sums and stores 3350 cycles).
constexpr int kSumWarps = 8;
constexpr int kSplitThreads = 32 * (2 + kSumWarps);

// Bytes of a row of a piece.  Its 16-byte chunk c lies at c ^ (tile row & 7), as in the 128-byte swizzle: eight lanes with the same chunk of
// eight rows, or with eight chunks of one row, hit distinct banks.
constexpr int kPitch = 32 * 4;

template <int BN>
struct SplitCfg {
    static constexpr int kStageBytes = BM * BK + BN * BK;
    static constexpr int kStages = BN == 64 ? 6 : BN == 128 ? 4 : 3;
    // Partial sums lie in pieces of 32 columns, [piece][row]: what goes to one CTA is contiguous and leaves as soon as a warp has staged it.
    static constexpr int kPieces = BN / 32;
    static constexpr int kRecvBytes = kPieces * (BM + kMaxSplit) * kPitch;   // C parts of up to ceil(128 / C) rows
    static constexpr int kTmemCols = BN == 192 ? 256 : BN;
    static constexpr int kSmemBytes = kStages * kStageBytes + kRecvBytes + BM * 4 + 1024 + 256;
    static_assert(kPieces * BM * kPitch <= kStages * kStageBytes, "the parts to be sent are staged over the operand stages");
};

// The cluster barrier without memory ordering: for "every CTA has got its parts", which the parts' own mbarriers have ordered.
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void prefetch_map(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}
__device__ __forceinline__ void dsmem_copy(uint32_t dst_cluster, uint32_t src, uint32_t bytes, uint32_t bar_cluster) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_cluster),
                 "r"(src), "r"(bytes), "r"(bar_cluster)
                 : "memory");
}

// OUT_F32 with p.gate: the gated residual, y += gate[col] * result.
template <int BN, int OUT>
__global__ void __launch_bounds__(kSplitThreads, 1)
convrot_gemm_splitk_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const GemmParams p) {
    using Cfg = SplitCfg<BN>;
    constexpr int S = Cfg::kStages;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    // layout: [S x (A tile | B tile), later the parts to be sent] [parts received] [scales] [barriers] [tmem slot] [abort flag]
    const uint32_t recv = smem_base + S * Cfg::kStageBytes;
    const uint32_t scales = recv + Cfg::kRecvBytes;               // act_scale of the rows this CTA finishes
    const uint32_t bars = scales + BM * 4;
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (S + s); };
    const uint32_t tfull_bar = bars + 8u * (2 * S), recv_bar = bars + 8u * (2 * S + 1);
    uint8_t *tail = smem_gen + S * Cfg::kStageBytes + Cfg::kRecvBytes + BM * 4 + 8 * (2 * S + 2);
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(tail);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tail + 8);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int rank = (int)cluster_ctarank();
    int C;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(C));
    const int m_tiles = (p.m + BM - 1) / BM;
    const int tile = blockIdx.x / C;
    const int m0 = (tile % m_tiles) * BM;
    const int n0 = (tile / m_tiles) * BN;
    const int k_blocks = p.k / BK;
    const int kb0 = k_blocks * rank / C, kb1 = k_blocks * (rank + 1) / C;
    const int rows = p.m - m0 < BM ? p.m - m0 : BM;              // of this tile
    auto row_begin = [&](int r) { return rows * r / C; };        // CTA r finishes rows row_begin(r) .. row_begin(r + 1) - 1
    const int my_begin = row_begin(rank), my_rows = row_begin(rank + 1) - my_begin;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(tfull_bar, 1);
        mbar_init(recv_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_arrive_expect_tx(recv_bar, (uint32_t)((C - 1) * my_rows * kPitch * Cfg::kPieces));
        prefetch_map(&tma_a);
        prefetch_map(&tma_b);
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
    cluster_arrive();   // waited for before the first part is sent: every CTA's barriers exist by then
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    tpb_grid_dep_launch();
    tpb_grid_dep_wait();

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            for (int kb = kb0; kb < kb1; kb++) {
                const int it = kb - kb0, s = it % S;
                if (!mbar_wait(empty_bar(s), ((it / S) & 1u) ^ 1u, abort_flag, p.status, (15u << 24) | s, true)) break;
                mbar_arrive_expect_tx(full_bar(s), Cfg::kStageBytes);
                const uint32_t a_dst = smem_base + s * Cfg::kStageBytes;
                tma_load_2d(a_dst, &tma_a, full_bar(s), kb * BK, m0);
                tma_load_2d(a_dst + BM * BK, &tma_b, full_bar(s), kb * BK, n0);
            }
        }
        __syncwarp();
        cluster_wait();
        cluster_arrive_relaxed();
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            const uint32_t idesc = make_idesc_i8<BN>(false);
            bool ok = true;
            for (int kb = kb0; kb < kb1; kb++) {
                const int it = kb - kb0, s = it % S;
                ok = mbar_wait(full_bar(s), (it / S) & 1u, abort_flag, p.status, (16u << 24) | s);
                if (!ok) break;
                tc_fence_after();
                const uint32_t a_addr = smem_base + s * Cfg::kStageBytes;
                const uint64_t a_desc = make_kmajor_sw128_desc(a_addr);
                const uint64_t b_desc = make_kmajor_sw128_desc(a_addr + BM * BK);
#pragma unroll
                for (int kk = 0; kk < BK / UMMA_K; kk++)
                    tc_mma_i8(tmem_base, a_desc + 2u * kk, b_desc + 2u * kk, idesc, (it > 0 || kk > 0) ? 1u : 0u);
                tc_commit(empty_bar(s));
            }
            if (ok) tc_commit(tfull_bar);
        }
        __syncwarp();
        cluster_wait();
        cluster_arrive_relaxed();
    } else {
        // ---------------- parts out, sums, epilogue ----------------
        const int quarter = warp & 3;
        // the columns that this thread finishes, and what it needs of them
        constexpr int kChunks = BN / 4, kRowStep = 32 * kSumWarps / kChunks, kBatch = 4;   // 192 columns: five rows at a time, 16 threads idle
        const int t = (int)threadIdx.x - 64;
        const int ch = t % kChunks, col = n0 + 4 * ch;
        const bool col_ok = t < kRowStep * kChunks && col < p.n;
        const size_t out_off = (size_t)(m0 + my_begin) * (size_t)p.ldy + (size_t)col;
        float4 ws = make_float4(0.f, 0.f, 0.f, 0.f), gt = ws;
        if (OUT != OUT_S32 && col_ok) {
            ws = __ldg(reinterpret_cast<const float4 *>(p.w_scale + col));
            if (OUT == OUT_F32 && p.gate != nullptr) gt = __ldcg(reinterpret_cast<const float4 *>(p.gate + col));
        }
        if (OUT != OUT_S32 && t < my_rows)
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(scales + 4u * (uint32_t)t), "f"(__ldcg(p.act_scale + m0 + my_begin + t)) : "memory");
        bool ok = mbar_wait(tfull_bar, 0, abort_flag, p.status, (17u << 24) | 1u, true);
        ok = __all_sync(0xffffffffu, ok);
        cluster_wait();
        if (ok) {
            tc_fence_after();
            const int q0 = quarter * 32;
            const int row = q0 + lane;
            if (q0 < rows) {
                // every MMA has read its operands: the operand stages now hold the parts to be sent;
                // this CTA's own part goes straight among the received ones
                const bool mine = row >= my_begin && row < my_begin + my_rows;
                const uint32_t dst = mine ? recv + (uint32_t)((rank * Cfg::kPieces * my_rows + row - my_begin) * kPitch)
                                          : smem_base + (uint32_t)(row * kPitch);
                const uint32_t dst_step = (uint32_t)((mine ? my_rows : BM) * kPitch);
                // this warp's rows that CTA `lane` finishes
                const int begin = row_begin(lane), cnt = row_begin(lane + 1) - begin;
                const int lo = begin > q0 ? begin : q0;
                const int hi = begin + cnt < q0 + 32 ? begin + cnt : q0 + 32;
                const bool sends = lane < C && lane != rank && lo < hi;
                const uint32_t to = sends ? mapa(recv + (uint32_t)((rank * Cfg::kPieces * cnt + lo - begin) * kPitch), (uint32_t)lane) : 0u;
                const uint32_t to_bar = sends ? mapa(recv_bar, (uint32_t)lane) : 0u;
                const uint32_t sw = (uint32_t)(row & 7);
                const uint32_t t_row = tmem_base + ((uint32_t)q0 << 16);
                constexpr int kMine = Cfg::kPieces / 2;      // of a warp: one half of its quarter's columns
                const int c0 = (warp - 2) / 4 * kMine;
                uint32_t r[2][32];
                tc_ld_32x32(t_row + (uint32_t)(c0 * 32), r[0]);
#pragma unroll
                for (int i = 0; i < kMine; i++) {
                    const int c = c0 + i;
                    uint32_t(&v)[32] = r[i & 1];
                    tc_wait_ld_dep(v);
                    if (i + 1 < kMine) tc_ld_32x32(t_row + (uint32_t)((c + 1) * 32), r[(i + 1) & 1]);
#pragma unroll
                    for (int g = 0; g < 8; g++)
                        st_shared_v4(dst + (uint32_t)c * dst_step + (((uint32_t)g ^ sw) << 4), v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (sends)
                        dsmem_copy(to + (uint32_t)(c * cnt * kPitch), smem_base + (uint32_t)((c * BM + lo) * kPitch),
                                   (uint32_t)((hi - lo) * kPitch), to_bar);
                    __syncwarp();
                }
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kSumWarps) : "memory");   // this CTA's own part and the scales are in place
        if (ok) {
            ok = mbar_wait(recv_bar, 0, abort_flag, p.status, (17u << 24) | 2u, true);
            ok = __all_sync(0xffffffffu, ok);
        }
        cluster_arrive_relaxed();   // this warp has seen every part arrive (or has given up)
        if (ok) {
            // A thread keeps its four columns and takes every kRowStep-th row, kBatch of them at a time with all their loads in flight.
#pragma unroll 1
            for (int lr0 = t / kChunks; lr0 < my_rows && col_ok; lr0 += kBatch * kRowStep) {
                float as[kBatch];
                float4 xv[kBatch];
                int4 a[kBatch];
#pragma unroll
                for (int b = 0; b < kBatch; b++) {
                    const int lr = lr0 + b * kRowStep;
                    a[b] = make_int4(0, 0, 0, 0);
                    as[b] = 0.0f;
                    xv[b] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (lr < my_rows && OUT != OUT_S32) {
                        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(as[b]) : "r"(scales + 4u * (uint32_t)lr));
                        if (OUT == OUT_F32 && p.gate != nullptr)
                            xv[b] = __ldcg(reinterpret_cast<const float4 *>(static_cast<const float *>(p.y) + out_off + (size_t)lr * (size_t)p.ldy));
                    }
                }
                // (a row past the last reads the last one's: the loads stay one batch, without branches between them)
                uint32_t at[kBatch];
#pragma unroll
                for (int b = 0; b < kBatch; b++) {
                    const int lr = min(lr0 + b * kRowStep, my_rows - 1);
                    at[b] = (uint32_t)(((ch >> 3) * my_rows + lr) * kPitch) + ((uint32_t)((ch & 7) ^ ((my_begin + lr) & 7)) << 4);
                }
                const uint8_t *src = smem_gen + (recv - smem_base);
#pragma unroll 2
                for (int r = 0; r < C; r++, src += Cfg::kPieces * my_rows * kPitch) {
                    int4 v[kBatch];
#pragma unroll
                    for (int b = 0; b < kBatch; b++) v[b] = *reinterpret_cast<const int4 *>(src + at[b]);
#pragma unroll
                    for (int b = 0; b < kBatch; b++) {
                        a[b].x += v[b].x; a[b].y += v[b].y; a[b].z += v[b].z; a[b].w += v[b].w;
                    }
                }
#pragma unroll
                for (int b = 0; b < kBatch; b++) {
                    const int lr = lr0 + b * kRowStep;
                    if (lr >= my_rows) break;
                    const size_t off = out_off + (size_t)lr * (size_t)p.ldy;
                    if (OUT == OUT_S32) {
                        *reinterpret_cast<int4 *>(static_cast<int32_t *>(p.y) + off) = a[b];
                        continue;
                    }
                    float4 v = make_float4(__fmul_rn(__fmul_rn(__int2float_rn(a[b].x), as[b]), ws.x), __fmul_rn(__fmul_rn(__int2float_rn(a[b].y), as[b]), ws.y),
                                           __fmul_rn(__fmul_rn(__int2float_rn(a[b].z), as[b]), ws.z), __fmul_rn(__fmul_rn(__int2float_rn(a[b].w), as[b]), ws.w));
                    if (OUT == OUT_F32) {
                        if (p.gate != nullptr)
                            v = make_float4(__fmaf_rn(gt.x, v.x, xv[b].x), __fmaf_rn(gt.y, v.y, xv[b].y), __fmaf_rn(gt.z, v.z, xv[b].z),
                                            __fmaf_rn(gt.w, v.w, xv[b].w));
                        *reinterpret_cast<float4 *>(static_cast<float *>(p.y) + off) = v;
                    } else {
                        const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
                        *reinterpret_cast<uint2 *>(static_cast<__nv_bfloat16 *>(p.y) + off) =
                            make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
                    }
                }
            }
        }
    }

    // ---------------- teardown ----------------
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        // A role gave up.  Give copies and MMAs still in flight time to land before shared memory and TMEM are released.
        for (int i = 0; i < 200; i++) __nanosleep(1000);
        __syncthreads();
    }
    cluster_wait();   // every part that this CTA sent has arrived: its receiver waited for it
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(Cfg::kTmemCols) : "memory");
    }
}

template <int BN, int OUT>
int launch_split(tpb_handle_t h, cudaStream_t st, const GemmParams &p, const int8_t *q, const void *w8, int split) {
    using Cfg = SplitCfg<BN>;
    CUtensorMap ma, mb;
    int rc = make_kmajor_map(h, &ma, q, p.m, p.k, BM);
    if (rc != TPB_OK) return rc;
    rc = make_kmajor_map(h, &mb, w8, p.n, p.k, BN);
    if (rc != TPB_OK) return rc;
    auto kern = convrot_gemm_splitk_kernel<BN, OUT>;
    static tpb_per_device_once smem_set;
    TPB_CUDA(h, tpb_set_max_smem_once(h, kern, Cfg::kSmemBytes, smem_set));
    const int64_t tiles = (int64_t)((p.m + BM - 1) / BM) * ((p.n + BN - 1) / BN);
    TPB_CUDA(h, tpb_launch_pdl_cluster(kern, dim3((unsigned)(tiles * split)), dim3(kSplitThreads), Cfg::kSmemBytes, st, split, ma, mb, p));
    return TPB_OK;
}

template <int BN>
int launch_split_out(tpb_handle_t h, cudaStream_t st, const GemmParams &p, int y_dtype, const int8_t *q, const void *w8, int split) {
    switch (y_dtype) {
        case TPB_F32: return launch_split<BN, OUT_F32>(h, st, p, q, w8, split);
        case TPB_BF16: return launch_split<BN, OUT_BF16>(h, st, p, q, w8, split);
        case TPB_S32: return launch_split<BN, OUT_S32>(h, st, p, q, w8, split);
    }
    return tpb_fail(h, TPB_ERR_INVALID_ARG, "gemm: unsupported y_dtype %d", y_dtype);
}

// How many clusters of `parts` CTAs the device holds at once.
int max_clusters(int parts) {
    auto kern = convrot_gemm_splitk_kernel<192, OUT_F32>;      // every variant takes most of an SM's shared memory: one CTA per SM
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(parts * 256));
    cfg.blockDim = dim3(kSplitThreads);
    cfg.dynamicSmemBytes = SplitCfg<192>::kSmemBytes;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)parts;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitCfg<192>::kSmemBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

}  // namespace

// Fills the handle's table of cluster counts (its device is current): SMs come in groups whose sizes differ from one device to the next, so three CTAs to
// a cluster are 45 clusters on one with 148 SMs, four 33, eight 15.  0 where it cannot be told: K is then not split so.
void tpb_gemm_splitk_init(tpb_handle_t h) {
    for (int parts = 2; parts <= kMaxSplit; parts++) h->max_clusters[parts] = max_clusters(parts);
}

// bn = 64, 128 or 192 columns per tile; split = 2 .. 8 CTAs per tile, at most p.k / 128.
int tpb_launch_gemm_splitk(tpb_handle_t h, cudaStream_t st, const tpb_gemm::GemmParams &p, int y_dtype, const int8_t *q, const void *w8,
                           int bn, int split) {
    switch (bn) {
        case 64: return launch_split_out<64>(h, st, p, y_dtype, q, w8, split);
        case 128: return launch_split_out<128>(h, st, p, y_dtype, q, w8, split);
        default: return launch_split_out<192>(h, st, p, y_dtype, q, w8, split);
    }
}
